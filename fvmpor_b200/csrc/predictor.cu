// Learned Newton initial iterate: a per-node MLP 8 -> 64 -> 64 -> 64 -> 1
// with GELU, BF16 weights and activations, FP32 accumulation on the sm_100a
// tensor cores (tcgen05.mma, accumulators in TMEM), trained on the device
// with hand-written forward and backward kernels and Adam.
//
// The reference has no counterpart (its Newton iterate is IDAS's BDF
// predictor).  The network's iterate is judged by the FP64 nonlinear
// residual: on every step where it is tried, y_pred + w * MLP(x) is kept
// only if its residual norm is below the BDF predictor's, otherwise the
// plain BDF extrapolation is used.
//
// Tile shape: a CTA owns a tile of 128 nodes; node r is TMEM lane r, and a
// node's 64 hidden values are shared by two threads (inference) or four
// (training): warp w works on lanes 32 (w % 4) .. + 31 and on the columns of
// its group w / 4.  One elected thread issues the MMAs (M = 128, N = 64, K = 16
// per instruction; the first layer pads its 8 inputs to K = 16), commits them
// to an mbarrier, and all threads read the FP32 accumulators back with
// tcgen05.ld for the bias + GELU epilogue, which writes the next layer's BF16
// operand straight into shared memory.  Backward: dA = dZ W (the forward
// weight tile read as an MN-major operand) and the weight gradients
// dW += dZ^T A (both operands read MN-major, accumulated in TMEM over the
// CTA's tiles) run on the tensor cores; the CTAs' gradients are summed in a
// fixed order by the kernel that takes the Adam step.
#include "predictor.cuh"
#include "krylov.cuh"
#include "reduce.cuh"
#include "tc05.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace fvmb {

using namespace tc05;

constexpr int kTile = 128;
// bf16 operand layouts inside the packed weight buffer (in 16-bit units)
constexpr int kW1s = 0;                       // 64 x 16
constexpr int kW2s = kW1s + kMlpH * kMlpK0;   // 64 x 64
constexpr int kW3s = kW2s + kMlpH * kMlpH;    // 64 x 64
constexpr int kWsz = kW3s + kMlpH * kMlpH;    // 9216 halves = 18432 B

// floats of a CTA's partial gradient: the parameters and the loss, 16-byte rows
constexpr int kPartial = (kNTrain + 1 + 3) & ~3;
static_assert(kOffW2 % 4 == 0 && kOffW3 % 4 == 0, "vector stores of the weights' gradients");

constexpr uint32_t kIdescFwd = idesc_bf16_f32(128, 64, false, false);
constexpr uint32_t kIdescBwd = idesc_bf16_f32(128, 64, false, true);

struct Predictor {
    DevBuf<float> p;          // [kNParam] FP32 master parameters
    DevBuf<float> m, v;       // Adam moments
    DevBuf<unsigned short> wl;
    DevBuf<float> partial;    // per-CTA gradients [nblk][kPartial]
    DevBuf<float> gsum;       // [kNTrain + 1] (last = loss sum)
    DevBuf<float> X, out;     // features / network output for all nodes
    DevBuf<double> yg, ypg, Fg;
    DevBuf<float> losses;     // loss sum of each batch of an epoch
    // error flag in mapped host memory: kernels write it only on a timeout, the
    // host reads it after its wait for the stream, without a copy
    struct Flag {
        int *h = nullptr, *p = nullptr;
        Flag() {
            FVM_CUDA(cudaHostAlloc(&h, sizeof(int), cudaHostAllocMapped));
            *h = 0;
            FVM_CUDA(cudaHostGetDevicePointer(&p, h, 0));
        }
        ~Flag() { cudaFreeHost(h); }
        Flag(const Flag&) = delete;
        Flag& operator=(const Flag&) = delete;
    } err;
    long adam_t = 0;
    bool ready = false;
};

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
// with the derivative d/dx [x Phi(x)] = Phi(x) + x phi(x)
__device__ __forceinline__ float gelu_and_grad(float x, float& grad) {
    const float u = 1.0f + erff(x * 0.70710678118654752f);
    grad = 0.5f * u + x * (0.39894228040143268f * __expf(-0.5f * x * x));
    return 0.5f * x * u;
}

// The same function by the normal tail Phi(-a) = exp(-a^2 / 2) t P(t),
// t = 1 / (1 + 0.28 a), a = |x|: the form of Hastings' approximations (Abramowitz
// & Stegun 7.1.25-26), with six coefficients fitted here by least squares,
// reweighted towards the minimax of the weighted tail (5.4e-9): two MUFU
// operations and nine multiply-adds.  In FP32 its largest error on [-8, 8] is
// 3.8e-7 and the root mean square 6.1e-8, against 4.5e-7 and 6.8e-8 of gelu();
// infinities and NaN give what gelu() gives.  Only for the last hidden layer of
// inference, whose values stay in FP32: the layers before it round to BF16,
// where a last-bit difference turns into one of 2^-8 near a tie.
__device__ __forceinline__ float gelu_tail(float x) {
    float t, e;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(fabsf(x), 0.28f, 1.0f)));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * x * -0.72134752f));
    float r = -0.10703232884407043f;
    r = fmaf(r, t, 0.39492541551589966f);
    r = fmaf(r, t, -0.24527788162231445f);
    r = fmaf(r, t, 0.2756578326225281f);
    r = fmaf(r, t, 0.06476791948080063f);
    r = fmaf(r, t, 0.11695902049541473f);
    const float q = t * e * r;
    return x * (x < 0.0f ? q : 1.0f - q);
}
__device__ __forceinline__ unsigned short bf16_bits(float x) {
    __nv_bfloat16 b = __float2bfloat16_rn(x);
    return *reinterpret_cast<unsigned short*>(&b);
}
// a in the low half
__device__ __forceinline__ uint32_t bf16_pair(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// FP32 masters -> BF16 operand tiles
__global__ void k_pack_weights(const float* __restrict__ P, unsigned short* __restrict__ wl) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < kMlpH * kMlpK0) {
        int n = t / kMlpK0, k = t % kMlpK0;
        float v = k < kMlpIn ? P[kOffW1 + n * kMlpIn + k] : 0.0f;
        wl[kW1s + il_off(n, k, kMlpK0) / 2] = bf16_bits(v);
    }
    if (t < kMlpH * kMlpH) {
        int n = t / kMlpH, k = t % kMlpH;
        wl[kW2s + il_off(n, k, kMlpH) / 2] = bf16_bits(P[kOffW2 + n * kMlpH + k]);
        wl[kW3s + il_off(n, k, kMlpH) / 2] = bf16_bits(P[kOffW3 + n * kMlpH + k]);
    }
}

constexpr int kFwdThreads = 256, kTrainThreads = 512;

// shared-memory carve-up common to the forward and training kernels
struct MlpSmem {
    unsigned short* W;   // packed weight tiles
    unsigned short* A0;  // 128 x 16
    unsigned short* A1;  // 128 x 64
    unsigned short* A2;  // 128 x 64 (training)
    unsigned short* Za;  // 128 x 64 (training): dZ of layers 3 and 1
    unsigned short* Zb;  // 128 x 64 (training): dZ of layer 2
    float* prm;          // b1, b2, b3, w4, b4, mu, sd (FP32 copies)
    float* sout;         // [column groups][128] shares of the output layer's sum
    float* red;          // [4][258] per-warp column sums (training)
    uint64_t* bar;
    uint32_t* tbase;
};

constexpr int kPrmB1 = 0, kPrmB2 = 64, kPrmB3 = 128, kPrmW4 = 192, kPrmB4 = 256, kPrmMu = 260, kPrmSd = 268,
              kPrmN = 276;
constexpr int kRedN = 258;

__host__ __device__ constexpr size_t mlp_smem_bytes(bool train) {
    return (size_t)kWsz * 2 + 128 * 16 * 2 + (train ? 4 : 1) * 128 * 64 * 2 + kPrmN * 4 +
           (train ? 4 * 128 + 4 * kRedN : 2 * 128) * 4 + 32;
}

__device__ MlpSmem carve(unsigned char* base, bool train) {
    MlpSmem s;
    unsigned char* p = base;
    s.W = (unsigned short*)p; p += kWsz * 2;
    s.A0 = (unsigned short*)p; p += 128 * 16 * 2;
    s.A1 = (unsigned short*)p; p += 128 * 64 * 2;
    s.A2 = s.Za = s.Zb = nullptr;
    if (train) {
        s.A2 = (unsigned short*)p; p += 128 * 64 * 2;
        s.Za = (unsigned short*)p; p += 128 * 64 * 2;
        s.Zb = (unsigned short*)p; p += 128 * 64 * 2;
    }
    // the weight-gradient MMAs read up to 1 KB past Za and Zb (issue_wgrad)
    s.prm = (float*)p; p += kPrmN * 4;
    s.sout = (float*)p; p += (train ? 4 : 2) * 128 * 4;
    s.red = (float*)p; p += train ? 4 * kRedN * 4 : 0;
    s.bar = (uint64_t*)p; p += 16;
    s.tbase = (uint32_t*)p;
    return s;
}
static_assert((kPrmN * 4) % 16 == 0 && (4 * kRedN * 4) % 16 == 0 && kPrmN * 4 >= 1024, "carve()");

__device__ void load_params(const MlpSmem& s, const float* __restrict__ P, const unsigned short* __restrict__ wl) {
    const uint4* src = reinterpret_cast<const uint4*>(wl);
    uint4* dst = reinterpret_cast<uint4*>(s.W);
    for (int i = threadIdx.x; i < kWsz * 2 / 16; i += blockDim.x) dst[i] = src[i];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        const int k = i & 63;
        s.prm[i] = P[i < 64 ? kOffB1 + k : i < 128 ? kOffB2 + k : i < 192 ? kOffB3 + k : kOffW4 + k];
    }
    if (threadIdx.x == 0) s.prm[kPrmB4] = P[kOffB4];
    if (threadIdx.x < 8) {
        s.prm[kPrmMu + threadIdx.x] = P[kOffMu + threadIdx.x];
        float sd = P[kOffSd + threadIdx.x];
        s.prm[kPrmSd + threadIdx.x] = sd > 0.0f ? sd : 1.0f;
    }
    // the padding of the first layer's operand
    if (threadIdx.x < 128)
        *reinterpret_cast<uint4*>((unsigned char*)s.A0 + il_off(threadIdx.x, 8, 16)) = make_uint4(0, 0, 0, 0);
}

// raw features of row0 + threadIdx.x / 2 (four per thread, the first 256
// threads), zeros past row n
__device__ __forceinline__ float4 load_features(const float* __restrict__ X, long row0, long n) {
    const long row = row0 + (threadIdx.x >> 1);
    return threadIdx.x < 256 && row < n ? reinterpret_cast<const float4*>(X)[2 * row + (threadIdx.x & 1)]
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
}
// normalised into the layer-1 operand
__device__ __forceinline__ void write_features(const MlpSmem& s, float4 f, long row0, long n) {
    if (threadIdx.x >= 256) return;
    const int r = threadIdx.x >> 1, k = 4 * (threadIdx.x & 1);
    uint2 h = make_uint2(0u, 0u);
    if (row0 + r < n) {
        const float *mu = s.prm + kPrmMu + k, *sd = s.prm + kPrmSd + k;
        h = make_uint2(bf16_pair((f.x - mu[0]) / sd[0], (f.y - mu[1]) / sd[1]),
                       bf16_pair((f.z - mu[2]) / sd[2], (f.w - mu[3]) / sd[3]));
    }
    *reinterpret_cast<uint2*>((unsigned char*)s.A0 + il_off(r, k, 16)) = h;
}

// eight values of a row into columns [c, c + 8) of a 128 x 64 operand
__device__ __forceinline__ void store8(unsigned short* dst, int r, int c, const float* v) {
    *reinterpret_cast<uint4*>((unsigned char*)dst + il_off(r, c, 64)) =
        make_uint4(bf16_pair(v[0], v[1]), bf16_pair(v[2], v[3]), bf16_pair(v[4], v[5]), bf16_pair(v[6], v[7]));
}

// this thread's row of the tile and its accumulators' TMEM address
__device__ __forceinline__ int tile_row() { return threadIdx.x & 127; }
__device__ __forceinline__ uint32_t lane_addr(uint32_t tmem, int col) {
    return tmem + ((threadIdx.x & 96u) << 16) + col;
}

// bias + GELU epilogue of a hidden layer: columns [c0, c0 + NC) of this
// thread's TMEM lane -> BF16 row of `dst`
template <int NC>
__device__ __forceinline__ void epilogue_hidden(uint32_t tmem, int c0, const float* bias, unsigned short* dst) {
    float v[NC];
    tmem_ld<NC>(lane_addr(tmem, c0), v);
#pragma unroll
    for (int c = 0; c < NC; c += 8) {
        float g[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) g[j] = gelu(v[c + j] + bias[c0 + c + j]);
        store8(dst, tile_row(), c0 + c, g);
    }
}

// one layer of MMAs: D(tmem col) = A (128 x K, K-major) x W (64 x K)^T
__device__ void issue_layer(uint32_t dtm, const unsigned short* A, const unsigned short* W, int K) {
    uint32_t a = smem_u32(A), b = smem_u32(W);
    for (int s = 0; s < K / 16; ++s)
        mma_bf16(dtm, smem_desc(a + s * 256, 128, K * 16), smem_desc(b + s * 256, 128, K * 16), kIdescFwd, s > 0);
}

struct Phase {
    uint32_t ph = 0;
};

// waits for the MMAs committed by thread 0; false (and the error flag) on timeout
__device__ bool sync_mma(const MlpSmem& s, Phase& ph, int* err) {
    bool ok = mbar_wait(s.bar, ph.ph & 1u);
    if (!ok) {
        atomicExch(err, 1);
        ok = mbar_wait(s.bar, ph.ph & 1u);   // give in-flight work a second bounded chance
    }
    ph.ph++;
    fence_after_sync();
    // every thread leaves with the same verdict, so the tile loop stays uniform
    return __syncthreads_and(ok ? 1 : 0) != 0;
}

__device__ void commit_from_thread0(const MlpSmem& s) {
    if (threadIdx.x == 0) mma_commit(s.bar);
}

// ------------------------------------------------------------------ inference
// Bound by the GELUs (41 M of them for the 214k nodes of the headline box), so
// the tiles' epilogues have to fill the SM: two threads per node and four CTAs
// per SM, whose MMA waits and barriers hide behind each other's epilogues.
// 214,221 rows, one B200, the whole call: 102.9 us with one thread per node,
// erff for all three layers and the error flag copied back, 59.6 us like this.
__global__ void __launch_bounds__(kFwdThreads, 4) k_mlp_forward(const float* __restrict__ X, long n,
                                                     const float* __restrict__ P,
                                                     const unsigned short* __restrict__ wl,
                                                     float* __restrict__ out, int* err) {
    extern __shared__ __align__(128) unsigned char smem[];
    MlpSmem s = carve(smem, false);
    const long ntiles = (n + kTile - 1) / kTile;
    float4 f = load_features(X, (long)blockIdx.x * kTile, n);
    load_params(s, P, wl);
    if (threadIdx.x < 32) tmem_alloc(s.tbase, 64);
    if (threadIdx.x == 0) {
        mbar_init(s.bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *s.tbase;
    constexpr int NC = 32;
    const int c0 = NC * (threadIdx.x >> 7);
    Phase ph;
    bool ok = true;
    for (long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
        write_features(s, f, tile * kTile, n);
        f = load_features(X, (tile + gridDim.x) * kTile, n);   // the next tile's, on their way meanwhile
        fence_smem_async();
        __syncthreads();
        if (threadIdx.x == 0) {
            fence_after_sync();
            issue_layer(tmem, s.A0, s.W + kW1s, 16);
        }
        commit_from_thread0(s);
        ok = sync_mma(s, ph, err);
        epilogue_hidden<NC>(tmem, c0, s.prm + kPrmB1, s.A1);
        fence_before_sync();
        fence_smem_async();
        __syncthreads();
        if (threadIdx.x == 0) {
            fence_after_sync();
            issue_layer(tmem, s.A1, s.W + kW2s, 64);
        }
        commit_from_thread0(s);
        ok = sync_mma(s, ph, err) && ok;
        epilogue_hidden<NC>(tmem, c0, s.prm + kPrmB2, s.A1);
        fence_before_sync();
        fence_smem_async();
        __syncthreads();
        if (threadIdx.x == 0) {
            fence_after_sync();
            issue_layer(tmem, s.A1, s.W + kW3s, 64);
        }
        commit_from_thread0(s);
        ok = sync_mma(s, ph, err) && ok;
        // output layer on the CUDA cores: y = gelu(z3 + b3) . w4 + b4
        float acc = 0.0f;
        {
            float v[NC];
            tmem_ld<NC>(lane_addr(tmem, c0), v);
            const float *b3 = s.prm + kPrmB3 + c0, *w4 = s.prm + kPrmW4 + c0;
#pragma unroll
            for (int j = 0; j < NC; ++j) acc = fmaf(gelu_tail(v[j] + b3[j]), w4[j], acc);
        }
        s.sout[threadIdx.x] = acc;
        fence_before_sync();
        __syncthreads();
        const long row = tile * kTile + threadIdx.x;
        if (threadIdx.x < kTile && row < n)
            out[row] = s.prm[kPrmB4] + (s.sout[threadIdx.x] + s.sout[kTile + threadIdx.x]);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        fence_after_sync();
        tmem_dealloc(tmem, 64);
    }
}

// ------------------------------------------------------------------ training
// sums of 16 columns over the warp's 32 rows by a transposing butterfly: each
// exchange hands the partner the half of the columns it keeps, so after
// offsets 16, 8, 4, 2 a lane holds one column (col_of_lane) summed over 16
// rows, and offset 1 completes it; 16 exchanges instead of 5 per column
__device__ __forceinline__ int col_of_lane() {
    const int l = threadIdx.x & 31;
    return ((l >> 1) & 1) | (((l >> 2) & 1) << 1) | (((l >> 3) & 1) << 2) | (((l >> 4) & 1) << 3);
}
__device__ __forceinline__ float col_sum16(float (&v)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int o = 16 >> s, c = 16 >> (s + 1);
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < c; ++j) {
            const float send = up ? v[j] : v[j + c], mine = up ? v[j + c] : v[j];
            v[j] = mine + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// dA(tmem dcol) = dZ (128 x 64, K-major) x W (64 x 64 weight tile read as the
// MN-major operand of W^T)
__device__ void issue_backward(uint32_t dtm, const unsigned short* dZ, const unsigned short* W) {
    uint32_t a = smem_u32(dZ), b = smem_u32(W);
    for (int s2 = 0; s2 < 4; ++s2)
        mma_bf16(dtm, smem_desc(a + s2 * 256, 128, 1024), smem_desc(b + s2 * 2048, 1024, 128), kIdescBwd, s2 > 0);
}

// dW(tmem, row o at lane o) += dZ^T A over the tile's 128 rows, A 128 x K: both
// tiles read as MN-major operands, 16 rows per instruction.  M is 128 although
// dZ has 64 columns: lanes 64.. get products of what follows in shared memory
// (the next row group, past the last one the 1 KB after the tile) and are
// never read.
__device__ void issue_wgrad(uint32_t dtm, const unsigned short* dZ, const unsigned short* A, int K, bool first) {
    const uint32_t a = smem_u32(dZ), b = smem_u32(A);
    const uint32_t idesc = idesc_bf16_f32(128, K, true, true);
    for (int s = 0; s < 8; ++s)
        mma_bf16(dtm, smem_desc(a + s * 2048, 1024, 128), smem_desc(b + s * 32 * K, 16 * K, 128), idesc,
                 !first || s > 0);
}

// one pass over rows [begin, end) of (X, Y): loss = mean (mlp(x) - y)^2;
// writes this CTA's gradient (scaled by 1/count) and loss sum to partial.
// A batch has fewer tiles than the chip has room for, so the chain of one
// tile counts: four threads per row, the GELU and its derivative formed
// together (the derivatives stay in registers for the way back), weight
// gradients on the tensor cores, bias sums in registers until the end.  An
// epoch of 65,536 rows in batches of 8,192 took 1,137 us with one thread per
// row, the weight gradients on the CUDA cores and a wait for the loss after each
// batch; 203 us like this (whole call, one B200).
__global__ void __launch_bounds__(kTrainThreads, 1) k_mlp_train(const float* __restrict__ X, const float* __restrict__ Y,
                                                      long begin, long end, long tiles_per_cta,
                                                      const float* __restrict__ P,
                                                      const unsigned short* __restrict__ wl,
                                                      float* __restrict__ partial, int* err) {
    extern __shared__ __align__(128) unsigned char smem[];
    MlpSmem s = carve(smem, true);
    if (threadIdx.x < 32) tmem_alloc(s.tbase, 256);
    if (threadIdx.x == 0) {
        mbar_init(s.bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    // the samples do not come from the kernel ahead (the last batch's step; an
    // epoch's first batch has none, train_pass), the parameters do
    const long first = (long)blockIdx.x * tiles_per_cta;
    float4 f = load_features(X, begin + first * kTile, end);
    pdl_wait_and_trigger();
    load_params(s, P, wl);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *s.tbase;
    const uint32_t D = tmem, W3 = tmem + 64, W2 = tmem + 128, W1 = tmem + 192;
    const float inv_count = 1.0f / (float)max(1l, end - begin);
    Phase ph;
    bool ok = true;
    constexpr int NC = 16;
    const int r = tile_row(), cg = threadIdx.x >> 7, c0 = NC * cg;
    float sum_b1 = 0.f, sum_b2 = 0.f, sum_b3 = 0.f, sum_w4 = 0.f, sum_b4 = 0.f, loss = 0.f;
    // forward epilogue of a hidden layer, keeping the derivatives
    auto hidden = [&](const float* bias, unsigned short* dst, float (&dg)[NC]) {
        float v[NC];
        tmem_ld<NC>(lane_addr(D, c0), v);
#pragma unroll
        for (int j = 0; j < NC; ++j) v[j] = gelu_and_grad(v[j] + bias[c0 + j], dg[j]);
        store8(dst, r, c0, v);
        store8(dst, r, c0 + 8, v + 8);
        fence_before_sync();
        fence_smem_async();
        __syncthreads();
    };
    // backward epilogue: dz = dA gelu'(z) in place of dg
    auto backward = [&](unsigned short* dZ, float (&dg)[NC]) {
        float v[NC];
        tmem_ld<NC>(lane_addr(D, c0), v);
#pragma unroll
        for (int j = 0; j < NC; ++j) dg[j] *= v[j];
        store8(dZ, r, c0, dg);
        store8(dZ, r, c0 + 8, dg + 8);
        fence_before_sync();
        fence_smem_async();
        __syncthreads();
    };
    for (long t = 0; t < tiles_per_cta && ok; ++t) {
        const long row0 = begin + (first + t) * kTile, row = row0 + r;
        const bool valid = row < end;
        const float target = valid ? Y[row] : 0.0f;
        float dg1[NC], dg2[NC], dg3[NC], h3[NC];
        // ---- forward
        write_features(s, f, row0, end);
        if (t + 1 < tiles_per_cta) f = load_features(X, row0 + kTile, end);
        fence_smem_async();
        __syncthreads();
        if (threadIdx.x == 0) { fence_after_sync(); issue_layer(D, s.A0, s.W + kW1s, 16); }
        commit_from_thread0(s);
        ok = sync_mma(s, ph, err) && ok;
        hidden(s.prm + kPrmB1, s.A1, dg1);
        if (threadIdx.x == 0) { fence_after_sync(); issue_layer(D, s.A1, s.W + kW2s, 64); }
        commit_from_thread0(s);
        ok = sync_mma(s, ph, err) && ok;
        hidden(s.prm + kPrmB2, s.A2, dg2);
        if (threadIdx.x == 0) { fence_after_sync(); issue_layer(D, s.A2, s.W + kW3s, 64); }
        commit_from_thread0(s);
        ok = sync_mma(s, ph, err) && ok;
        {
            float v[NC], acc = 0.0f;
            tmem_ld<NC>(lane_addr(D, c0), v);
            const float *b3 = s.prm + kPrmB3 + c0, *w4 = s.prm + kPrmW4 + c0;
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                h3[j] = gelu_and_grad(v[j] + b3[j], dg3[j]);
                acc = fmaf(h3[j], w4[j], acc);
            }
            s.sout[threadIdx.x] = acc;
        }
        __syncthreads();
        const float outv = s.prm[kPrmB4] + ((s.sout[r] + s.sout[128 + r]) + (s.sout[256 + r] + s.sout[384 + r]));
        const float e = valid ? outv - target : 0.0f;
        const float dout = 2.0f * e * inv_count;
        // ---- layer 3
#pragma unroll
        for (int j = 0; j < NC; ++j) dg3[j] *= dout * s.prm[kPrmW4 + c0 + j];
        store8(s.Za, r, c0, dg3);
        store8(s.Za, r, c0 + 8, dg3 + 8);
        fence_before_sync();
        fence_smem_async();
        __syncthreads();
        if (threadIdx.x == 0) { fence_after_sync(); issue_backward(D, s.Za, s.W + kW3s); }
        commit_from_thread0(s);
        if (threadIdx.x == 0) issue_wgrad(W3, s.Za, s.A2, 64, t == 0);
        sum_b3 += col_sum16(dg3);
        // ---- output layer gradients
        loss += e * e;
        sum_b4 += dout;
#pragma unroll
        for (int j = 0; j < NC; ++j) h3[j] *= dout;
        sum_w4 += col_sum16(h3);
        // ---- layer 2
        ok = sync_mma(s, ph, err) && ok;
        backward(s.Zb, dg2);
        if (threadIdx.x == 0) { fence_after_sync(); issue_backward(D, s.Zb, s.W + kW2s); }
        commit_from_thread0(s);
        if (threadIdx.x == 0) issue_wgrad(W2, s.Zb, s.A1, 64, t == 0);
        sum_b2 += col_sum16(dg2);
        // ---- layer 1 (the MMAs that read Za completed with the ones just
        // waited for: a commit covers all earlier ones)
        ok = sync_mma(s, ph, err) && ok;
        backward(s.Za, dg1);
        if (threadIdx.x == 0) { fence_after_sync(); issue_wgrad(W1, s.Za, s.A0, 16, t == 0); }
        commit_from_thread0(s);
        sum_b1 += col_sum16(dg1);
        ok = sync_mma(s, ph, err) && ok;
    }
    // the CTA's gradient: weights from TMEM (rows at lanes 0..63), bias sums
    // over the four row groups
    float* g = partial + (size_t)blockIdx.x * kPartial;
    auto store = [&](float* dst, const float* v, int n) {
#pragma unroll
        for (int j = 0; j < n; j += 4)
            *reinterpret_cast<float4*>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    };
    const int q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
    if (q < 2) {
        float v[NC];
        tmem_ld<NC>(lane_addr(W3, c0), v);
        store(g + kOffW3 + r * 64 + c0, v, NC);
        tmem_ld<NC>(lane_addr(W2, c0), v);
        store(g + kOffW2 + r * 64 + c0, v, NC);
        if (cg == 0) {
            tmem_ld<NC>(lane_addr(W1, 0), v);
            store(g + kOffW1 + r * kMlpIn, v, kMlpIn);
        }
    }
    float* red = s.red + q * kRedN;
    if (!(lane & 1)) {
        const int c = c0 + col_of_lane();
        red[c] = sum_b1;
        red[64 + c] = sum_b2;
        red[128 + c] = sum_b3;
        red[192 + c] = sum_w4;
    }
    if (cg == 0) {
        sum_b4 = warp_sum(sum_b4);
        loss = warp_sum(loss);
        if (lane == 0) {
            red[256] = sum_b4;
            red[257] = loss;
        }
    }
    fence_before_sync();
    __syncthreads();
    for (int j = threadIdx.x; j < kRedN; j += blockDim.x) {
        const float t = ((s.red[j] + s.red[kRedN + j]) + s.red[2 * kRedN + j]) + s.red[3 * kRedN + j];
        const int k = j & 63;
        g[j < 64 ? kOffB1 + k : j < 128 ? kOffB2 + k : j < 192 ? kOffB3 + k : j < 256 ? kOffW4 + k
          : j == 256 ? kOffB4 : kNTrain] = t;
    }
    if (threadIdx.x < 32) {
        fence_after_sync();
        tmem_dealloc(tmem, 256);
    }
}

// Sums the CTAs' gradients in a fixed order (kSumGroups runs of consecutive
// CTAs, each in CTA order, then the runs in order) and, given the parameters, takes the
// Adam step and rewrites the weight's BF16 operand.  32 parameters per CTA, so
// that the loads of a run are coalesced and all of a parameter's in flight.
constexpr int kSumGroups = 8;
struct AdamArgs {
    float lr, b1, b2, eps, bc1, bc2;
    float *P, *m, *v;
    unsigned short* wl;
    float* loss;   // the batch's loss sum, or nullptr
};
__global__ void __launch_bounds__(32 * kSumGroups) k_grad_step(const float* __restrict__ partial, int nblk,
                                                               float* __restrict__ g, AdamArgs a) {
    pdl_wait_and_trigger();
    __shared__ float part[kSumGroups][32];
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5, j = 32 * blockIdx.x + lane;
    const int per = (nblk + kSumGroups - 1) / kSumGroups, b1 = min(nblk, (grp + 1) * per);
    float s = 0.0f;
    if (j <= kNTrain) {
#pragma unroll 8
        for (int b = grp * per; b < b1; ++b) s += partial[(size_t)b * kPartial + j];
    }
    part[grp][lane] = s;
    __syncthreads();
    if (grp || j > kNTrain) return;
    float gj = 0.0f;
#pragma unroll
    for (int k = 0; k < kSumGroups; ++k) gj += part[k][lane];
    g[j] = gj;
    if (!a.P) return;
    if (j == kNTrain) {
        if (a.loss) *a.loss = gj;
        return;
    }
    const float mj = a.b1 * a.m[j] + (1.0f - a.b1) * gj;
    const float vj = a.b2 * a.v[j] + (1.0f - a.b2) * gj * gj;
    a.m[j] = mj;
    a.v[j] = vj;
    const float w = a.P[j] - a.lr * (mj / a.bc1) / (sqrtf(vj / a.bc2) + a.eps);
    a.P[j] = w;
    if (j < kOffB1) a.wl[kW1s + il_off(j / kMlpIn, j % kMlpIn, kMlpK0) / 2] = bf16_bits(w);
    else if (j >= kOffW2 && j < kOffB2)
        a.wl[kW2s + il_off((j - kOffW2) / kMlpH, (j - kOffW2) % kMlpH, kMlpH) / 2] = bf16_bits(w);
    else if (j >= kOffW3 && j < kOffB3)
        a.wl[kW3s + il_off((j - kOffW3) / kMlpH, (j - kOffW3) % kMlpH, kMlpH) / 2] = bf16_bits(w);
}

// ------------------------------------------------------------------ features
__global__ void k_features(int N, const double* __restrict__ h_n, const double* __restrict__ h_prev,
                           const double* __restrict__ ypred, float ldt, const float* __restrict__ statf,
                           float* __restrict__ X) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    double h = h_n[i];
    float4 a = make_float4((float)h, (float)(h - h_prev[i]), (float)(ypred[i] - h), ldt);
    float4 b = make_float4(statf[i], statf[(size_t)N + i], statf[(size_t)2 * N + i], 0.0f);
    float4* x4 = reinterpret_cast<float4*>(X + (size_t)i * 8);
    x4[0] = a;
    x4[1] = b;
}

// guess = y_pred + w * mlp on free rows; y' follows the corrector relation
__global__ void k_apply_guess(int N, const float* __restrict__ out, const double* __restrict__ ypred,
                              const double* __restrict__ yppred, const double* __restrict__ h_n,
                              const unsigned char* __restrict__ ntype, double rtol, double atol, double cj,
                              double* __restrict__ yg, double* __restrict__ ypg) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    double d = ntype[i] ? 0.0 : (rtol * fabs(h_n[i]) + atol) * (double)out[i];
    yg[i] = ypred[i] + d;
    ypg[i] = yppred[i] + cj * d;
}

// y = y_pred + a (y_guess - y_pred), y' likewise; e = y - y_pred
__global__ void k_take_guess(int N, double a, const double* __restrict__ yg, const double* __restrict__ ypg,
                             const double* __restrict__ ypred, const double* __restrict__ yppred,
                             double* __restrict__ y, double* __restrict__ yp, double* __restrict__ e) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const double d = a == 1.0 ? yg[i] - ypred[i] : a * (yg[i] - ypred[i]);
    y[i] = a == 1.0 ? yg[i] : ypred[i] + d;
    yp[i] = a == 1.0 ? ypg[i] : yppred[i] + a * (ypg[i] - yppred[i]);
    e[i] = d;
}

// out = (F0.F0, F0.F1, F1.F1), fixed-order reduction
__global__ void k_dot3(int N, const double* __restrict__ F0, const double* __restrict__ F1, double* partial,
                       unsigned* counter, double* out) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < N; k += gridDim.x * blockDim.x) {
        const double a = F0[k], b = F1[k];
        s0 += a * a;
        s1 += a * b;
        s2 += b * b;
    }
    __shared__ double red[3][32];
    s0 = warp_sum(s0);
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (lane == 0) { red[0][w] = s0; red[1][w] = s1; red[2][w] = s2; }
    __syncthreads();
    if (w < 3) {
        double t = lane < nw ? red[w][lane] : 0.0;
        t = warp_sum(t);
        if (lane == 0) partial[(size_t)blockIdx.x * 3 + w] = t;
    }
    last_block_reduce(partial, 3, counter, out);
}

__global__ void k_record(int N, int stride, int offset, const float* __restrict__ Xall,
                         const double* __restrict__ y_new, const double* __restrict__ ypred,
                         const double* __restrict__ h_n, const unsigned char* __restrict__ ntype, double rtol,
                         double atol, long base, long cap, float* __restrict__ X, float* __restrict__ Y) {
    long q = blockIdx.x * (long)blockDim.x + threadIdx.x;
    long i = offset + q * stride;
    if (i >= N) return;
    long slot = base + q;
    if (slot >= cap) return;
    for (int k = 0; k < 8; ++k) X[slot * 8 + k] = Xall[i * 8 + k];
    double w = rtol * fabs(h_n[i]) + atol;
    Y[slot] = ntype[i] ? 0.0f : (float)((y_new[i] - ypred[i]) / w);
}

// ------------------------------------------------------------------ host side
Predictor* predictor_get(fvm_ctx* c) {
    if (!c->pred) {
        Predictor* p = new Predictor();
        p->p.alloc(kNParam);
        p->m.alloc(kNTrain);
        p->v.alloc(kNTrain);
        p->wl.alloc(kWsz);
        p->gsum.alloc(kNTrain + 1);
        p->losses.alloc(4096);
        p->m.zero(c->stream);
        p->v.zero(c->stream);
        p->X.alloc((size_t)c->N * 8);
        p->out.alloc(c->N);
        p->yg.alloc(c->N);
        p->ypg.alloc(c->N);
        p->Fg.alloc(c->N);
        c->pred = p;
        raise_smem_limit(k_mlp_forward, mlp_smem_bytes(false));
        raise_smem_limit(k_mlp_train, mlp_smem_bytes(true));
    }
    return c->pred;
}

Predictor* predictor_of(fvm_ctx* c) { return (c->pred && c->pred->ready) ? c->pred : nullptr; }
bool predictor_ready(Predictor* p) { return p && p->ready; }

static void pack(fvm_ctx* c, Predictor* p) {
    fvm_launch(c, k_pack_weights, (kMlpH * kMlpH + 255) / 256, 256, 0, c->stream, p->p.p, p->wl.p);
}

void predictor_features(fvm_ctx* c, const double* h_n, const double* h_prev, const double* ypred, double dt,
                        float* X) {
    fvm_launch(c, k_features, grid_for(c->N, 256), 256, 0, c->stream, c->N, h_n, h_prev, ypred,
               (float)std::log10(std::max(dt, 1e-30)), c->statf.p, X);
}

void predictor_forward(fvm_ctx* c, Predictor* p, const float* X, int n, float* out) {
    long ntiles = ((long)n + kTile - 1) / kTile;
    int grid = (int)std::min<long>(ntiles, 148 * 4);
    if (grid < 1) return;
    fvm_launch(c, k_mlp_forward, grid, kFwdThreads, mlp_smem_bytes(false), c->stream, X, (long)n, p->p.p, p->wl.p, out,
               p->err.p);
}

// squared residual-norm ratio below which the learned iterate is kept
constexpr double kGuessKeep = 0.25;

bool predictor_apply(fvm_ctx* c, Predictor* p, double rtol, double atol, double dt, double cj, const double* h_n,
                     const double* h_prev, const double* ypred, const double* yppred, double* y, double* yp,
                     double* e, double* F) {
    const int N = c->N;
    c->tm.begin(TM_PRED, c->stream);
    struct EndTimer {
        fvm_ctx* c;
        ~EndTimer() { c->tm.end(TM_PRED, c->stream); }
    } end_timer{c};
    c->tm.begin(TM_MLP, c->stream);
    predictor_features(c, h_n, h_prev, ypred, dt, p->X.p);
    predictor_forward(c, p, p->X.p, N, p->out.p);
    c->tm.end(TM_MLP, c->stream);
    fvm_launch(c, k_apply_guess, grid_for(N, 256), 256, 0, c->stream, N, p->out.p, ypred, yppred, h_n, c->ntype.p,
               rtol, atol, cj, p->yg.p, p->ypg.p);
    Perturb none;
    launch_residual(c, p->yg.p, p->ypg.p, none, nullptr, p->Fg.p);
    launch_residual(c, ypred, yppred, none, nullptr, F);
    // The residual is close to linear over one Newton correction, so along
    // y(a) = y_pred + a (y_guess - y_pred) its squared norm is the quadratic
    // through F0 = F(y_pred) and F1 = F(y_guess):
    //   |F(a)|^2 ~ A + 2a (B - A) + a^2 (A - 2B + C),  A = F0.F0, B = F0.F1, C = F1.F1.
    // Take its minimiser on [0, 1]; keep the BDF predictor when the learned
    // direction does not lower the residual.
    Krylov* K = krylov_scratch(c);
    fvm_launch(c, k_dot3, kRedBlocks, kRedThreads, 0, c->stream, N, F, p->Fg.p, K->partial.p, K->counter.p,
               K->res.p);
    FVM_CUDA(cudaMemcpyAsync(K->host, K->res.p, 3 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    ctx_sync(c);
    const double A = K->host[0], B = K->host[1], Cc = K->host[2];
    const double curv = A - 2.0 * B + Cc;   // |F1 - F0|^2
    if (!std::isfinite(A) || !std::isfinite(Cc) || !(curv > 0.0)) return false;
    double a = (A - B) / curv;
    a = std::min(1.0, a);
    const double pred = A + 2.0 * a * (B - A) + a * a * curv;
    // A learned start that lowers the residual only a little leaves Newton
    // converging (within its tolerance) to a point biased toward the guess,
    // which inflates the BDF error estimate: on the 3D benchmark, accepting
    // guesses at a 2 % residual drop raised the step count by 16 %.  Keep
    // the guess only when it halves the residual norm.
    if (!(a > 0.05) || !(pred < kGuessKeep * A)) return false;
    fvm_launch(c, k_take_guess, grid_for(N, 256), 256, 0, c->stream, N, a, p->yg.p, p->ypg.p, ypred, yppred, y, yp,
               e);
    if (a == 1.0) FVM_CUDA(cudaMemcpyAsync(F, p->Fg.p, sizeof(double) * N, cudaMemcpyDeviceToDevice, c->stream));
    else launch_residual(c, y, yp, none, nullptr, F);
    return true;
}

void recorder_push(fvm_ctx* c, Recorder* r, const float* Xall, const double* y_new, const double* ypred,
                   const double* h_n, double rtol, double atol) {
    if (!r || r->count >= r->cap) return;
    int offset = (int)(r->step % r->stride);
    long q = (c->N - offset + r->stride - 1) / r->stride;
    q = std::min(q, r->cap - r->count);
    if (q > 0)
        fvm_launch(c, k_record, grid_for(q, 256), 256, 0, c->stream, c->N, r->stride, offset, Xall, y_new, ypred, h_n,
                   c->ntype.p, rtol, atol, r->count, r->cap, r->X, r->Y);
    r->count += q;
    r->step++;
}

// gradient of the rows [begin, end) and, where the step names the parameters, one Adam
// step; chained: the kernel ahead on the stream is another batch's step (else
// it may be the one that writes X, which the training kernel reads early)
static void train_pass(fvm_ctx* c, Predictor* p, const float* X, const float* Y, long begin, long end, AdamArgs step,
                       bool chained) {
    long ntiles = (end - begin + kTile - 1) / kTile;
    int nblk = (int)std::min<long>(ntiles, 148);
    long per = (ntiles + nblk - 1) / nblk;
    nblk = (int)((ntiles + per - 1) / per);
    if ((long)p->partial.n < (long)nblk * kPartial) p->partial.alloc((size_t)nblk * kPartial);
    auto launch = [&](auto&&... args) {
        if (chained) fvm_launch_pdl(c, k_mlp_train, nblk, kTrainThreads, mlp_smem_bytes(true), c->stream, args...);
        else fvm_launch(c, k_mlp_train, nblk, kTrainThreads, mlp_smem_bytes(true), c->stream, args...);
    };
    launch(X, Y, begin, end, per, p->p.p, p->wl.p, p->partial.p, p->err.p);
    fvm_launch_pdl(c, k_grad_step, (kNTrain + 32) / 32, 32 * kSumGroups, 0, c->stream, p->partial.p, nblk, p->gsum.p,
                   step);
}

static int check_err(fvm_ctx* c, Predictor* p) {
    FVM_CUDA(cudaStreamSynchronize(c->stream));
    return *(volatile int*)p->err.h;
}

} // namespace fvmb

using namespace fvmb;

void fvmb_destroy_predictor(fvmb::Predictor* p) { delete p; }

#define API_TRY try {
#define API_CATCH                        \
    }                                    \
    catch (const Error& ex) {            \
        set_error(ex.what());            \
        return ex.code;                  \
    }                                    \
    catch (const std::exception& ex) {   \
        set_error(ex.what());            \
        return -1;                       \
    }

extern "C" int fvm_mlp_nparams(void) { return kNParam; }

extern "C" int fvm_mlp_set_params(fvm_ctx* c, const float* params_host) {
    API_TRY
    if (!c || !params_host) throw Error("fvm_mlp_set_params: null argument");
    Predictor* p = predictor_get(c);
    FVM_CUDA(cudaMemcpyAsync(p->p.p, params_host, sizeof(float) * kNParam, cudaMemcpyHostToDevice, c->stream));
    pack(c, p);
    p->m.zero(c->stream);
    p->v.zero(c->stream);
    p->adam_t = 0;
    p->ready = true;
    FVM_CUDA(cudaStreamSynchronize(c->stream));
    return 0;
    API_CATCH
}

extern "C" int fvm_mlp_get_params(fvm_ctx* c, float* params_host) {
    API_TRY
    if (!c || !params_host || !c->pred) throw Error("fvm_mlp_get_params: no predictor");
    FVM_CUDA(cudaMemcpyAsync(params_host, c->pred->p.p, sizeof(float) * kNParam, cudaMemcpyDeviceToHost, c->stream));
    FVM_CUDA(cudaStreamSynchronize(c->stream));
    return 0;
    API_CATCH
}

extern "C" int fvm_mlp_forward(fvm_ctx* c, const float* X, int n, float* out) {
    API_TRY
    if (!c || !X || !out || !c->pred) throw Error("fvm_mlp_forward: no predictor or null argument");
    predictor_forward(c, c->pred, X, n, out);
    FVM_CUDA(cudaGetLastError());
    int e = check_err(c, c->pred);
    return e ? 2 : 0;
    API_CATCH
}

extern "C" int fvm_mlp_grad(fvm_ctx* c, const float* X, const float* Y, int n, float* grad_host,
                            float* loss) {
    API_TRY
    if (!c || !X || !Y || !c->pred) throw Error("fvm_mlp_grad: no predictor or null argument");
    train_pass(c, c->pred, X, Y, 0, n, AdamArgs{}, false);
    std::vector<float> g(kNTrain + 1);
    FVM_CUDA(cudaMemcpyAsync(g.data(), c->pred->gsum.p, sizeof(float) * (kNTrain + 1), cudaMemcpyDeviceToHost,
                             c->stream));
    int e = check_err(c, c->pred);
    if (grad_host) std::copy(g.begin(), g.begin() + kNTrain, grad_host);
    if (loss) *loss = g[kNTrain] / std::max(1, n);
    return e ? 2 : 0;
    API_CATCH
}

extern "C" int fvm_mlp_train(fvm_ctx* c, const float* X, const float* Y, int n, int epochs, int batch, float lr,
                             float* loss_history) {
    API_TRY
    if (!c || !X || !Y || !c->pred || n <= 0 || epochs <= 0) throw Error("fvm_mlp_train: bad argument");
    Predictor* p = c->pred;
    if (batch <= 0) batch = 148 * 2 * kTile;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const long nbatch = ((long)n + batch - 1) / batch;
    std::vector<float> loss(nbatch);
    if ((long)p->losses.n < nbatch) p->losses.alloc(nbatch);
    for (int ep = 0; ep < epochs; ++ep) {
        for (long b0 = 0; b0 < n; b0 += batch) {
            p->adam_t++;
            const float bc1 = 1.0f - std::pow(b1, (float)p->adam_t), bc2 = 1.0f - std::pow(b2, (float)p->adam_t);
            train_pass(c, p, X, Y, b0, std::min<long>(n, b0 + batch),
                       AdamArgs{lr, b1, b2, eps, bc1, bc2, p->p.p, p->m.p, p->v.p, p->wl.p, p->losses.p + b0 / batch},
                       b0 > 0);
        }
        FVM_CUDA(cudaMemcpyAsync(loss.data(), p->losses.p, sizeof(float) * nbatch, cudaMemcpyDeviceToHost, c->stream));
        FVM_CUDA(cudaStreamSynchronize(c->stream));
        double lsum = 0.0;
        for (float l : loss) lsum += l;
        if (loss_history) loss_history[ep] = (float)(lsum / n);
    }
    p->ready = true;
    return check_err(c, p) ? 2 : 0;
    API_CATCH
}
