// One GMRES cycle in one persistent cooperative launch, for the assembled
// Krylov operator (fvm_opts.krylov_operator = 1) with the FP32 block-ILU(0)
// factor and FP32 basis.
//
// The Arnoldi step of decomp/gmres.c:412-511 (left-preconditioned and scaled
// by D = diag(ewt), as IDAS SPGMR runs it, ida_integrator.h:248-254) is
//   w = D P^-1 J D^-1 V_j,  CGS2 against V_0..V_j,  Givens update
// (linalg_dense.c:128-173).  With J assembled (the preconditioner set-up's
// difference-quotient Jacobian, shifted exactly to the current cj), every
// part of a step is local to the rows of one ILU block except the operator's
// reads of the direction at neighbouring nodes and the orthogonalisation's
// dot products.  So one CTA owns one ILU block for the whole cycle:
//   - its factor window and metadata are brought into shared memory ONCE per
//     cycle by bulk copies (the staged apply reloads them on every apply);
//   - per step it has the direction at its own nodes from its last basis pass,
//     gathers it at its halo nodes into shared memory, forms its rows of J t from there (rows in factor order,
//     one warp per 32 rows, entry-major slices with 16-bit local columns)
//     straight into the shared-memory vector the triangular sweeps work on,
//     runs both sweeps there, scales by ewt, and
//     orthogonalises its rows (by delayed reorthogonalisation in two passes
//     over the basis, or by CGS2 in three; row quads, fixed-order reductions
//     through per-block partials);
//   - every block computes the Hessenberg column, the rotations and the
//     stopping test from the same reduced numbers, so all take the same
//     decision without another barrier; block 0 keeps them and at the end
//     does the back substitution.
// One bounded grid barrier per step with delayed reorthogonalisation, two
// with CGS2 (after each dot pass).  The next
// direction is published block by block: a block raises its flag once its
// rows are written, and a block starting the next step waits (bounded) only
// for the flags of the blocks its operator rows reach, plus its two
// neighbours in node order.  Nothing returns to the host until the cycle
// ends.  Replaces, for this operator, the five launches per step of the
// difference-quotient path (node pass, element pass, gather, apply, CGS2).
#include "cgs.cuh"
#include "ilu.cuh"
#include "krylov.cuh"

#include <algorithm>
#include <cmath>

namespace fvmb {

struct FusedArgs {
    int N, m, nr_max, nh_max, halo_max;
    int nqp;                   // quads per block row array in shared memory (quad-transposed, quad_pos)
    size_t stage_max;          // shared bytes of the largest block's staged factor
    ArnState* st;
    double tol, sqrtN;         // stop when |g_j| / sqrt(N) <= tol
    double* coef;              // the solution's coefficients (times the scales), for k_combine_dev
    float* U;
    size_t ld;
    double* scale;
    float* tdir;               // D^-1 V_j, FP32, node order (read at neighbours)
    const double* ewt;
    const int* slptr;          // [slices + 1] first entry of each slice
    const int* blksl;          // [nb + 1] first slice of each block
    const unsigned short* op_lcol;   // entry -> index in the block's node list
    const int* halo_ptr;       // [nb + 1] the block's node list: its rows and halo
    const int* halo_node;
    const int* nbr_ptr;        // [nb + 1] blocks whose flags a block waits for
    const int* nbr;
    unsigned* flags;           // [nb] base + last step whose direction rows a block wrote
    unsigned* sync;            // arrival counter of the grid barriers
    unsigned base;             // above every flag of earlier launches
    const float* op_val;
    const float* op_dg;        // [N], factor order: ahh(h + d) on free rows, else 0
    float dcj;                 // cj - cj of the set-up
    const int* bstart;
    const IluBlk* blk;
    const unsigned short* lu_col;
    const unsigned short* meta;
    const float* lu;
    const int* lu_row;
    const double* beta2;       // ||D P^-1 r||^2 of the cycle's start
    double* partial;
    int* err;
    double* H;
};

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned atom_add_release_gpu(unsigned* p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// Grid barrier of the cycle on a counter that only grows (a launch leaves it at a
// multiple of the grid size, fused_cycle): a block adds 1 with release semantics
// and waits (acquire, bounded) until the counter reaches the next multiple
// of the grid size.  Its own arrival number says which multiple, so there is
// no generation word, no reset and no further step for the last block to
// arrive.  A block that gives up, or meets an error elsewhere, sets
// kSyncFail (above any count, fused_cycle): every block sees it at its next
// barrier and leaves, and err carries the reason to k_combine_dev.
constexpr unsigned kSyncFail = 1u << 30;
__device__ __forceinline__ void fused_fail(unsigned* sync, int* err, int code) {
    atomicExch(err, code);
    atomicOr(sync, kSyncFail);
}
__device__ __forceinline__ bool fused_sync(unsigned* sync, int* err, int* s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned old = atom_add_release_gpu(sync, 1u);
        bool ok = !(old & kSyncFail);
        if (ok) {
            const unsigned target = (old / gridDim.x + 1) * gridDim.x;
            long it = 0;
            unsigned v;
            while ((v = ld_acquire_gpu(sync)) < target) {
                if (++it > (1l << 26)) {
                    fused_fail(sync, err, 3);
                    break;
                }
            }
            ok = v >= target && !(v & kSyncFail);
        }
        *s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    return *s_ok != 0;
}

// the unrotated Hessenberg matrix by columns, c + 2 entries in column c: where
// column c starts
__host__ __device__ __forceinline__ int hess_words(int c) { return c * (c + 3) / 2; }

// barrier among `count` threads (whole warps) of the block on barrier `id`
__device__ __forceinline__ void named_barrier(int id, int count) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// One lane's row of an operator slice, up to 16 entries of it (longer rows read
// the rest in place).  Entries are stored four to a lane, so a slice is a few
// 16-byte loads of values and 8-byte loads of columns per lane: with single
// entries (24 loads of 4 and 2 bytes) the loads in flight took more registers
// and the operator 6.1 us per step on the 214k-node box instead of 4.9 (4.0
// with the directions in factor order, fused_prepare).
struct OpSlice {
    float4 v[4];
    uint2 c[4];
    float dg;
    int w;
};
constexpr int kOpGroup = 128;   // entries per group: four per lane
__device__ __forceinline__ void op_four(float& acc, const float* tl, const float4& v, const uint2& c) {
    acc = fmaf(v.x, tl[c.x & 0xffffu], acc);
    acc = fmaf(v.y, tl[c.x >> 16], acc);
    acc = fmaf(v.z, tl[c.y & 0xffffu], acc);
    acc = fmaf(v.w, tl[c.y >> 16], acc);
}

// the loads of slice sl (rows.x slices, rows.y the block's first row, rows.z
// rows; starts Sl): streamed once per step through L2 only, so that L1 keeps
// the block's basis rows between the passes.  All set before the conditional
// loads: see ilu_sweep
__device__ __forceinline__ void op_load(const FusedArgs& a, OpSlice& R, const int* Sl, const int3& rows, int sl,
                                        int lane) {
    R.w = 0;
    R.dg = 0.f;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        R.v[g] = make_float4(0.f, 0.f, 0.f, 0.f);
        R.c[g] = make_uint2(0u, 0u);
    }
    if (sl >= rows.x) return;
    const int base = Sl[sl];
    R.w = (Sl[sl + 1] - base) / kOpGroup;
    const float4* pv = reinterpret_cast<const float4*>(a.op_val + base) + lane;
    const uint2* pc = reinterpret_cast<const uint2*>(a.op_lcol + base) + lane;
#pragma unroll
    for (int g = 0; g < 4; ++g)
        if (g < R.w) {
            R.v[g] = __ldcg(pv + 32 * g);
            R.c[g] = __ldcg(pc + 32 * g);
        }
    R.dg = __ldcg(a.op_dg + rows.y + min(32 * sl + lane, rows.z - 1));
}
__device__ __forceinline__ void op_apply(const FusedArgs& a, const OpSlice& R, float* x, const float* tl,
                                         const int* Sl, const int3& rows, int sl, int lane) {
    if (sl >= rows.x) return;
    float acc = 0.f;
#pragma unroll
    for (int g = 0; g < 4; ++g)
        if (g < R.w) op_four(acc, tl, R.v[g], R.c[g]);
#pragma unroll 1
    for (int g = 4; g < R.w; ++g)
        op_four(acc, tl, __ldcg(reinterpret_cast<const float4*>(a.op_val + Sl[sl]) + lane + 32 * g),
                __ldcg(reinterpret_cast<const uint2*>(a.op_lcol + Sl[sl]) + lane + 32 * g));
    const int q = 32 * sl + lane;
    if (q < rows.z) x[q] = fmaf(-a.dcj * R.dg, tl[q], acc);
}

// Back substitution H y = g of the cycle's k columns (block 0), the coefficients
// times the basis vectors' scales to a.coef: the solution is formed without the
// host.  H comes back from global memory (this block wrote it) into the block's
// shared memory, whose other contents are no longer needed, packed by columns.
__host__ __device__ __forceinline__ int tri_words(int c) { return c * (c + 1) / 2; }
__device__ __forceinline__ void back_substitute(const FusedArgs& a, int k, const double* sc, const double* gs) {
    double* R = reinterpret_cast<double*>(ilu_smem());
    for (int e = threadIdx.x; e < k * k; e += blockDim.x) {
        const int i = e / k, c = e - i * k;
        if (i <= c) R[tri_words(c) + i] = __ldcg(a.H + (size_t)i * a.m + c);
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    // lane l holds rows l and l + 32
    double r0 = lane < k ? gs[lane] : 0.0, r1 = lane + 32 < k ? gs[lane + 32] : 0.0;
    for (int c = k - 1; c >= 0; --c) {
        const double* col = R + tri_words(c);
        const double d = col[c], top = __shfl_sync(0xffffffffu, c < 32 ? r0 : r1, c & 31);
        const double y = d != 0.0 ? top / d : 0.0;
        if (lane < c) r0 -= col[lane] * y;
        if (lane + 32 < c) r1 -= col[lane + 32] * y;
        if (lane == 0) a.coef[c] = y * sc[c];
    }
}

// at most 384 threads (one per row quad of a 1,536-row block; larger blocks
// loop), so a thread may hold up to 170 registers
constexpr int kFusedThreads = 384;

template <bool DEL, bool WIDE>
__global__ void __launch_bounds__(kFusedThreads, 1) k_arnoldi_fused(FusedArgs a) {
    // ca holds up to 2 (m + 1) + 2 reduced numbers on the delayed variant
    __shared__ double ca[DEL ? 132 : 64], cb[64], coef[64], sc[64], rc[64], rs[64], gs[64];
    // delayed variant: first projection of the pending column, t, p, H t and
    // the two combine coefficient sets
    __shared__ double hp[DEL ? 64 : 1], tv[DEL ? 64 : 1], pv[DEL ? 64 : 1], htv[DEL ? 64 : 1],
        c1[DEL ? 64 : 1], c2[DEL ? 64 : 1];
    // warp partials of the delayed variant's dot pass (two alternating groups)
    __shared__ double red[DEL ? 2 * (kFusedThreads / 32) * 2 * kCgsGroup : 1];
    __shared__ int s_done, s_ok;
    // the factor's place, read again for each sweep: held in registers through
    // the basis passes, which need them all, it would be spilled
    __shared__ IluShared<float> s_view;
    __shared__ int3 s_rows;   // operator slices, first row, rows
    unsigned char* const smem_raw = ilu_smem();
    const int b = blockIdx.x, nblk = gridDim.x;
    const int r0 = a.bstart[b], r1 = a.bstart[b + 1], nr = r1 - r0;
    const IluBlk B = a.blk[b];
    // staged factor (the layout of k_ilu_apply_smem), then the inverse of
    // the block's row order and its rows of W
    const IluStage<float> S(B, nr);
    float* x = S.x;
    uint64_t* mbar = S.bar;
    unsigned short* inv = reinterpret_cast<unsigned short*>(smem_raw + a.stage_max);
    // the block's rows of W (and of the pending vector), quad-transposed
    const int nqp = a.nqp;
    double* Ws = reinterpret_cast<double*>(smem_raw + a.stage_max + round16(2 * (size_t)a.nr_max));
    float* tl = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(Ws) + 32 * (size_t)nqp);
    // delayed variant: the block's rows of the pending vector v_k, then the
    // unrotated Hessenberg matrix (column c at Hs[hess_words(c) ..])
    double* Vs = reinterpret_cast<double*>(reinterpret_cast<unsigned char*>(tl) + round16(4 * (size_t)a.nh_max));
    double* Hs = Vs + 4 * (size_t)nqp;
    // delayed variant: the block's rows of ewt (quad-transposed, 1 in the
    // edge quads' padding), read by every step's scaling of W and of the
    // next direction instead of going to L2 for them
    double* Es = Hs + hess_words(a.m);
    // delayed variant: the halo's nodes, for the gather of every step's
    // direction there
    int* Hn = reinterpret_cast<int*>(Es + 4 * (size_t)nqp);
    // first entry of each of the block's operator slices
    int* Sl = DEL ? Hn + a.halo_max : reinterpret_cast<int*>(Vs);
    if (threadIdx.x == 0) {
        tc05::mbar_init(mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    __syncthreads();
    ilu_stage_bulk(S, B, nr, a.lu, a.lu_col, a.meta);
    if (threadIdx.x == 0) {
        x[nr] = 0.f;
        s_view = S.view(B);
        s_rows = make_int3(a.blksl[b + 1] - a.blksl[b], r0, nr);
    }
    for (int q = threadIdx.x; q < nr; q += blockDim.x) inv[a.lu_row[r0 + q] - r0] = (unsigned short)q;
    const int sl0 = a.blksl[b], nsl = a.blksl[b + 1] - sl0;
    const int h0 = a.halo_ptr[b], nh = a.halo_ptr[b + 1] - h0;
    for (int k = threadIdx.x; k <= nsl; k += blockDim.x) Sl[k] = a.slptr[sl0 + k];
    // the padding rows of the edge quads stay zero
    for (int k = threadIdx.x; k < 4 * nqp; k += blockDim.x) {
        Ws[k] = 0.0;
        if constexpr (DEL) {
            Vs[k] = 0.0;
            const int e = k / nqp, row = (r0 & ~3) + 4 * (k - e * nqp) + e;   // inverse of quad_pos
            Es[k] = row >= r0 && row < r1 ? a.ewt[row] : 1.0;
        }
    }
    if constexpr (DEL)
        for (int k = nr + threadIdx.x; k < nh; k += blockDim.x) Hn[k - nr] = a.halo_node[h0 + k];
    // All so far was there before the kernel ahead of this one, which wrote U_0
    // and its norm, could start: its launch need not have ended
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int m = a.m;
    const double tol = a.tol, sqrtN = a.sqrtN;
    // the cycle's initial residual norm (||D P^-1 r||, left by the host's
    // launches in a.beta2) decides whether any step is needed
    const double beta = sqrt(*a.beta2);
    const double rn0 = beta / sqrtN;
    for (int i = threadIdx.x; i <= m; i += blockDim.x) gs[i] = i == 0 ? beta : 0.0;
    // the scale of U_0 (1 / beta)
    const double s0 = beta > 0.0 ? 1.0 / beta : 0.0;
    if (threadIdx.x == 0) {
        sc[0] = s0;
        if (b == 0) {
            a.scale[0] = s0;
            a.st->done = 0;   // until the cycle ends
            a.st->j = 0;
        }
    }
    if (!isfinite(beta) || rn0 <= tol) {
        if (b == 0 && threadIdx.x == 0) {
            a.st->rnorm = rn0;
            a.st->j = 0;
            a.st->done = isfinite(beta) ? 1 : 3;
        }
        tc05::mbar_wait(mbar, 0);   // the factor copies land before the block leaves
        return;
    }
    bool ok = tc05::mbar_wait(mbar, 0);
    if (!ok) ok = tc05::mbar_wait(mbar, 0);   // copies in flight get a second bounded chance
    if (!__syncthreads_and(ok ? 1 : 0) && threadIdx.x == 0) fused_fail(a.sync, a.err, 2);   // all blocks stop at the next barrier
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    // vector-major partials: pa[v * nblk + b]
    double* pa = a.partial;
    double* pb = a.partial + (size_t)nblk * 64;
    // the block reads only basis rows that were complete before its last
    // barrier (its own rows; the other rows of its edge quads are masked
    // out and belong to blocks it waits for), so the read-only path is safe
    const BasisRows<float, false> UR{a.U, a.ld};
    const int q0 = r0 & ~3;
    const int nb0 = a.nbr_ptr[b], nb1 = a.nbr_ptr[b + 1];
    // step 0's direction s_0 U_0 / ewt at the block's own and halo nodes
    // (U_0 was written before the launch)
    for (int k = threadIdx.x; k < nh; k += blockDim.x) {
        const int node = a.halo_node[h0 + k];
        tl[k] = (float)(s0 * (double)__ldcg(a.U + node) / a.ewt[node]);
    }
    __syncthreads();
    for (int j = 0;; ++j) {
        const int nv = j + 1;
        // operator: x = J(cj) t for the block's rows, in factor order; a warp
        // keeps two slices in flight
        {
            const int lane = tid_here() & 31, first = tid_here() >> 5;
            OpSlice A, B;
            op_load(a, A, Sl, s_rows, first, lane);
            op_load(a, B, Sl, s_rows, first + nw, lane);
#pragma unroll 1
            for (int sl = first; sl < s_rows.x; sl += 2 * nw) {
                op_apply(a, A, x, tl, Sl, s_rows, sl, lane);
                op_load(a, A, Sl, s_rows, sl + 2 * nw, lane);
                op_apply(a, B, x, tl, Sl, s_rows, sl + nw, lane);
                op_load(a, B, Sl, s_rows, sl + 3 * nw, lane);
            }
        }
        __syncthreads();
        // preconditioner: both triangular sweeps in shared memory
        {
            const IluShared<float> V = s_view;
            ilu_sweep<float, false, WIDE>(V, 1, V.nl);
            ilu_sweep<float, true, WIDE>(V, 0, V.nu);
        }
        for (int k = threadIdx.x; k < nr; k += blockDim.x) {
            const int qp = quad_pos(r0, nqp, r0 + k);
            Ws[qp] = (DEL ? Es[qp] : a.ewt[r0 + k]) * (double)x[inv[k]];
        }
        __syncthreads();
        // Hessenberg column finalised by this step (-1: none yet), the entry
        // below its diagonal, and the scale of the basis vector it finalises
        int hcol = j;
        double hn = 0.0;
        double newscale = 0.0;
        if constexpr (!DEL) {
        // pass 1: a = U^T W
        block_dots_by_warp(a.U, a.ld, Ws, nqp, r0, r1, nv, false, ca);
        for (int i = threadIdx.x; i < nv; i += blockDim.x) pa[(size_t)i * nblk + b] = ca[i];
        if (!fused_sync(a.sync, a.err, &s_ok)) return;
        block_reduce_all_vmajor(pa, nv, nblk, ca);
        for (int i = threadIdx.x; i < nv; i += blockDim.x) coef[i] = ca[i] * sc[i] * sc[i];
        __syncthreads();
        // pass 2: W' = W - U diag(s^2) a; b = U^T W', ||W'||^2
        for (int r = q0 + 4 * threadIdx.x; r < r1; r += 4 * blockDim.x) {
            double acc[4];
            quad_combine(UR, coef, nv, r, acc);
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (r + e >= r0 && r + e < r1) Ws[quad_pos(r0, nqp, r + e)] -= acc[e];
        }
        __syncthreads();
        block_dots_by_warp(a.U, a.ld, Ws, nqp, r0, r1, nv, true, cb);
        for (int i = threadIdx.x; i <= nv; i += blockDim.x) pb[(size_t)i * nblk + b] = cb[i];
        if (!fused_sync(a.sync, a.err, &s_ok)) return;
        block_reduce_all_vmajor(pb, nv + 1, nblk, cb);
        double nrm2 = cb[nv];
        for (int i = 0; i < nv; ++i) {
            const double c = sc[i] * cb[i];
            nrm2 -= c * c;
        }
        nrm2 = nrm2 > 0.0 ? nrm2 : 0.0;
        const double snv = nrm2 > 0.0 ? 1.0 / sqrt(nrm2) : 0.0;
        for (int i = threadIdx.x; i < nv; i += blockDim.x) coef[i] = cb[i] * sc[i] * sc[i];
        __syncthreads();
        // pass 3: the new basis vector (unnormalised, scale snv) and the
        // next direction D^-1 V_{j+1}
        float* Un = a.U + a.ld * nv;
        for (int r = q0 + 4 * threadIdx.x; r < r1; r += 4 * blockDim.x) {
            double acc[4];
            quad_combine(UR, coef, nv, r, acc);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int k = r + e;
                if (k >= r0 && k < r1) {
                    const float u = (float)(Ws[quad_pos(r0, nqp, k)] - acc[e]);
                    Un[k] = u;
                    const float t = (float)(snv * (double)u / a.ewt[k]);
                    a.tdir[k] = t;
                    tl[inv[k - r0]] = t;
                }
            }
        }
        // the Hessenberg column of the two projections
        for (int i = threadIdx.x; i < nv; i += blockDim.x) ca[i] = sc[i] * (ca[i] + cb[i]);
        hn = sqrt(nrm2);
        newscale = snv;
        } else {
        // Delayed reorthogonalisation (DCGS2: Swirydowicz, Langou, Ananthan,
        // Yang & Thomas, Numer. Linear Algebra Appl. 28 (2021) e2343).  The
        // step's direction is v_k, the previous step's vector after one
        // projection; z = A v_k.  One pass over the basis gives
        // t = V^T v_k, p = V^T z, v_k.v_k and v_k.z, one grid barrier reduces
        // them.  Then q_k = (v_k - V t) / beta with beta^2 = v.v - t.t
        // finalises column k-1 of H (first projection of step k-1 plus t,
        // and beta below it); A q_k = (z - V_k H t) / beta by the Arnoldi
        // relation, so its first projection s and the next vector
        // v_{k+1} = A q_k - V_k s follow from the reduced numbers, and one
        // more pass over the basis writes both q_k (as U_k, scale 1/beta)
        // and v_{k+1}.  Two passes and one barrier per step instead of
        // four and two; the column of step k is final one step later.
        const int k = j;
        const int nbv = k == 0 ? 1 : k;   // basis vectors this step reads
        block_dots2_by_quad(a.U, a.ld, Vs, Ws, nqp, r0, r1, nbv, red, ca);
        const int nred = 2 * nbv + 2;
        for (int i = threadIdx.x; i < nred; i += blockDim.x) pa[(size_t)i * nblk + b] = ca[i];
        if (!fused_sync(a.sync, a.err, &s_ok)) return;
        block_reduce_all_vmajor(pa, nred, nblk, ca);
        double beta = 1.0, ck = 0.0;
        if (k == 0) {
            // v_1 = z - V_0 p_0
            if (threadIdx.x == 0) {
                const double p0 = sc[0] * ca[1];
                hp[0] = p0;
                c1[0] = 0.0;
                c2[0] = sc[0] * p0;
            }
            hcol = -1;
        } else {
            // four partial sums each: one chain of k dependent FP64
            // operations is a microsecond at the end of a cycle
            double t4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
            for (int i = 0; i < k; i += 4)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const double t = i + u < k ? sc[i + u] * ca[i + u] : 0.0;
                    t4[u] += t * t;
                }
            const double b2 = ca[2 * k] - ((t4[0] + t4[1]) + (t4[2] + t4[3]));
            beta = b2 > 0.0 ? sqrt(b2) : 0.0;
            for (int i = threadIdx.x; i <= k; i += blockDim.x) {
                const double t = i < k ? sc[i] * ca[i] : 0.0;
                tv[i] = t;
                pv[i] = i < k ? sc[i] * ca[k + i] : 0.0;
                Hs[hess_words(k - 1) + i] = i < k ? hp[i] + t : beta;
            }
            __syncthreads();
            // Ht = H[0..k][0..k-1] t (H[i][c] is zero below c + 1)
            for (int i = threadIdx.x; i <= k; i += blockDim.x) {
                double h4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
                for (int c = i > 0 ? i - 1 : 0; c < k; c += 4)
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (c + u < k) h4[u] += Hs[hess_words(c + u) + i] * tv[c + u];
                htv[i] = (h4[0] + h4[1]) + (h4[2] + h4[3]);
            }
            double p4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
            for (int i = 0; i < k; i += 4)
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (i + u < k) p4[u] += tv[i + u] * pv[i + u];
            const double tp = (p4[0] + p4[1]) + (p4[2] + p4[3]);
            __syncthreads();
            const double rb = beta > 0.0 ? 1.0 / beta : 0.0;
            const double sk = (ca[2 * k + 1] - tp - beta * htv[k]) * rb * rb;
            ck = htv[k] * rb + sk;
            for (int i = threadIdx.x; i < k; i += blockDim.x) {
                const double si = (pv[i] - htv[i]) * rb;
                c1[i] = sc[i] * tv[i];
                c2[i] = sc[i] * (htv[i] * rb + si - ck * tv[i] * rb);
                hp[i] = si;
            }
            if (threadIdx.x == 0) {
                hp[k] = sk;
                sc[k] = rb;
            }
            hcol = k - 1;
            hn = beta;
            newscale = rb;
        }
        __syncthreads();
        // q_k = v_k - V t (k >= 1), v_{k+1} = z / beta - (c_k / beta) v_k - V c2,
        // and the next direction D^-1 v_{k+1}
        {
            float* Uk = a.U + a.ld * k;
            const double rb = k == 0 ? 1.0 : (beta > 0.0 ? 1.0 / beta : 0.0);
            const double vcoef = k == 0 ? 0.0 : ck * rb;
            for (int r = q0 + 4 * threadIdx.x; r < r1; r += 4 * blockDim.x) {
                double acc1[4], acc2[4];
                quad_combine2(a.U, a.ld, c1, c2, nbv, r, acc1, acc2);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int q = r + e;
                    if (q >= r0 && q < r1) {
                        const int qp = quad_pos(r0, nqp, q);
                        const double vq = Vs[qp];
                        if (k >= 1) Uk[q] = (float)(vq - acc1[e]);
                        const double vn = Ws[qp] * rb - vcoef * vq - acc2[e];
                        Vs[qp] = vn;
                        const float t = (float)(vn / Es[qp]);
                        a.tdir[q] = t;
                        tl[inv[q - r0]] = t;
                    }
                }
            }
        }
        }
        // publish this block's rows of the next direction
        __syncthreads();
        if (threadIdx.x == 0) st_release_gpu(a.flags + b, a.base + (unsigned)nv);   // release: the block's writes before the barrier
        __syncthreads();
        // rotations and stopping test for the finalised column, the same in
        // every block (the same reduced numbers, the same operations), on
        // thread 0 while the other warps wait for the next direction's rows
        // this block reads (bounded) and gather them into shared memory
        if (warp > 0) {
            if (warp == 1) {
                for (int kk = nb0 + lane; kk < nb1; kk += 32) {
                    const unsigned* f = a.flags + a.nbr[kk];
                    long it = 0;
                    while (ld_acquire_gpu(f) < a.base + (unsigned)nv) {
                        if (++it > (1l << 26)) { fused_fail(a.sync, a.err, 3); break; }
                    }
                }
            }
            named_barrier(1, blockDim.x - 32);
            for (int kk = nr + threadIdx.x - 32; kk < nh; kk += blockDim.x - 32)
                tl[kk] = __ldcg(a.tdir + (DEL ? Hn[kk - nr] : a.halo_node[h0 + kk]));
        } else if (threadIdx.x == 0) {
            int done = 0;
            if (hcol >= 0) {
                double* hc = ca;
                if constexpr (DEL) {
                    for (int i = 0; i <= hcol; ++i) hc[i] = Hs[hess_words(hcol) + i];
                }
                hc[hcol + 1] = hn;
                if (!isfinite(hn) || !isfinite(hc[hcol])) {
                    done = 3;
                } else {
                    double cur = hc[0];
                    for (int i = 0; i < hcol; ++i) {
                        const double nx = hc[i + 1];
                        hc[i] = rc[i] * cur + rs[i] * nx;
                        cur = -rs[i] * cur + rc[i] * nx;
                    }
                    hc[hcol] = cur;
                    const double den = hypot(hc[hcol], hc[hcol + 1]);
                    double cj_, sj_;
                    if (den == 0.0) { cj_ = 1.0; sj_ = 0.0; }
                    else { cj_ = hc[hcol] / den; sj_ = hc[hcol + 1] / den; }
                    rc[hcol] = cj_;
                    rs[hcol] = sj_;
                    hc[hcol] = den;
                    const double gj = gs[hcol];
                    gs[hcol + 1] = -sj_ * gj;
                    gs[hcol] = cj_ * gj;
                    sc[hcol + 1] = newscale;
                    const double rn = fabs(gs[hcol + 1]) / sqrtN;
                    if (rn <= tol || hn == 0.0) done = 1;
                    else if (hcol + 1 == m) done = 2;
                    if (b == 0) {
                        for (int i = 0; i <= hcol; ++i) a.H[(size_t)i * m + hcol] = hc[i];
                        a.scale[hcol + 1] = newscale;
                        a.st->rnorm = rn;
                        a.st->j = hcol + 1;
                    }
                }
            }
            if (b == 0) a.st->done = done;
            s_done = done;
        }
        __syncthreads();
        if (s_done) {
            if (b == 0 && s_done != 3) back_substitute(a, hcol + 1, sc, gs);
            return;
        }
    }
}

static int fused_sync_slot(int nb) { return ((nb + 31) & ~31) + 32; }

using FusedKernel = void (*)(FusedArgs);
static FusedKernel fused_kernel(int variant, bool wide) {
    if (wide) return variant ? k_arnoldi_fused<true, true> : k_arnoldi_fused<false, true>;
    return variant ? k_arnoldi_fused<true, false> : k_arnoldi_fused<false, false>;
}

constexpr int kFusedMaxDim = 62;   // the reduced numbers' arrays

// Gram-Schmidt of the fused cycle on this context: 0 CGS2 (two projections,
// two grid barriers per step), 1 delayed reorthogonalisation (DCGS2)
static int fused_variant(const fvm_ctx* c) { return c->krylov_variant ? 1 : 0; }

// dynamic shared bytes of a cycle of up to m steps
static size_t fused_bytes(const BlockILU* P, int variant, int m) {
    const size_t cycle = variant ? P->fused_smem_d + 8 * (size_t)hess_words(m) : P->fused_smem;
    return std::max(cycle, 8 * (size_t)tri_words(m));   // (back_substitute)
}

// values of the operator's slices from the set-up's Jacobian (FP64 CSR) and
// the cj coefficient of its diagonal, in factor order
__global__ void k_op_refresh(long ne, const int* __restrict__ src, const double* __restrict__ J, float* __restrict__ v,
                             int N, const int* __restrict__ lu_row, const double* __restrict__ ahhp,
                             const unsigned char* __restrict__ ntype, float* __restrict__ dgq) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ne) {
        const int p = src[t];
        v[t] = p >= 0 ? (float)J[p] : 0.f;
    }
    if (t < N) {
        const int row = lu_row[t];
        dgq[t] = ntype[row] ? 0.f : (float)ahhp[row];
    }
}

// flags and barrier counter back to zero: first, after a failed launch (whose
// blocks left at different barriers), and before either could overflow
void fused_reset(fvm_ctx* c) {
    if (!c->ilu || !c->ilu->flags.n) return;
    c->ilu->flags.zero(c->stream);
    c->ilu->fused_launches = 0;
}

// Host side: the slice layout (once per pattern), the launch checks, and the
// per-set-up refresh.  Returns false when the fused cycle cannot run on this
// context (FP32 staged factor does not fit, or the blocks cannot all be
// resident at once); the caller then uses the separate kernels.
bool fused_prepare(fvm_ctx* c, int m) {
    BlockILU* P = c->ilu;
    // the cycle inlines the block-Jacobi apply; the Schur-coupled apply
    // runs as its own cooperative launch between the separate kernels
    if (!P || !P->built || P->factored != 1 || m > kFusedMaxDim || P->schur_iters >= 0) return false;
    cudaStream_t s = c->stream;
    if (!P->op_built) {
        P->op_built = true;
        P->fused_ok = false;
        const int nb = P->nb;
        if (!P->smem_stage[1]) return false;
        // a block's slices: entries' local columns and sources, slice starts; its
        // node list (its rows in factor order, then the other operator
        // columns, sorted) and the blocks owning those nodes.  A slice's rows
        // have one colour and are consecutive in factor order, and so are,
        // mostly, their neighbours of another colour: a warp's reads of the
        // direction hit few banks twice (in node order, eight lanes to a bank)
        struct Block {
            std::vector<int> start, src, nodes, nbr;
            std::vector<unsigned short> lcol;
        };
        std::vector<Block> block(nb);
        parallel_for(nb, std::max(1l, 1024l * nb / c->N), [&](long first, long last) {
            for (long b = first; b < last; ++b) {
                const int r0 = P->h_bstart[b], r1 = P->h_bstart[b + 1];
                Block& B = block[b];
                std::vector<int> col, halo;
                B.start.assign(1, 0);
                for (int q0 = r0; q0 < r1; q0 += 32) {
                    const int n = std::min(32, r1 - q0);
                    int width = 0;
                    for (int l = 0; l < n; ++l) {
                        const int row = P->h_lu_row[q0 + l];
                        width = std::max(width, P->h_rowptr[row + 1] - P->h_rowptr[row]);
                    }
                    width = (width + 3) & ~3;
                    const size_t base = col.size();
                    col.resize(base + 32 * (size_t)width);
                    B.src.resize(base + 32 * (size_t)width);
                    for (int l = 0; l < 32; ++l) {
                        const int row = l < n ? P->h_lu_row[q0 + l] : P->h_lu_row[q0];
                        const int p0 = P->h_rowptr[row], len = l < n ? P->h_rowptr[row + 1] - p0 : 0;
                        for (int k = 0; k < width; ++k) {
                            const size_t e = base + (size_t)kOpGroup * (k / 4) + 4 * l + k % 4;
                            col[e] = k < len ? P->h_col[p0 + k] : row;
                            B.src[e] = k < len ? p0 + k : -1;
                            if (col[e] < r0 || col[e] >= r1) halo.push_back(col[e]);
                        }
                    }
                    B.start.push_back((int)col.size());
                }
                std::sort(halo.begin(), halo.end());
                halo.erase(std::unique(halo.begin(), halo.end()), halo.end());
                B.nodes.assign(P->h_lu_row.begin() + r0, P->h_lu_row.begin() + r1);
                std::vector<int> place(r1 - r0);   // of the block's own nodes
                for (int q = r0; q < r1; ++q) place[P->h_lu_row[q] - r0] = q - r0;
                B.nodes.insert(B.nodes.end(), halo.begin(), halo.end());
                B.lcol.resize(col.size());
                for (size_t e = 0; e < col.size(); ++e)
                    B.lcol[e] = (unsigned short)(col[e] >= r0 && col[e] < r1
                                                     ? place[col[e] - r0]
                                                     : r1 - r0 + (std::lower_bound(halo.begin(), halo.end(), col[e]) -
                                                                  halo.begin()));
                if (b > 0) B.nbr.push_back((int)b - 1);
                if (b + 1 < nb) B.nbr.push_back((int)b + 1);
                for (int v : halo)
                    B.nbr.push_back((int)(std::upper_bound(P->h_bstart.begin(), P->h_bstart.end(), v) -
                                          P->h_bstart.begin()) - 1);
                std::sort(B.nbr.begin(), B.nbr.end());
                B.nbr.erase(std::unique(B.nbr.begin(), B.nbr.end()), B.nbr.end());
            }
        });
        std::vector<int> slptr(1, 0), blksl(1, 0), opsrc;
        std::vector<int> halo_ptr(1, 0), halo_node, nbr_ptr(1, 0), nbr;
        std::vector<unsigned short> lcol;
        int nr_max = 0, nh_max = 0, halo_max = 0;
        for (int b = 0; b < nb; ++b) {
            const Block& B = block[b];
            const int nr = P->h_bstart[b + 1] - P->h_bstart[b];
            if (B.nodes.size() >= 65535 || opsrc.size() + B.src.size() >= (size_t)INT32_MAX) return false;
            nr_max = std::max(nr_max, nr);
            nh_max = std::max(nh_max, (int)B.nodes.size());
            halo_max = std::max(halo_max, (int)B.nodes.size() - nr);
            for (size_t k = 1; k < B.start.size(); ++k) slptr.push_back((int)opsrc.size() + B.start[k]);
            blksl.push_back((int)slptr.size() - 1);
            opsrc.insert(opsrc.end(), B.src.begin(), B.src.end());
            lcol.insert(lcol.end(), B.lcol.begin(), B.lcol.end());
            nbr.insert(nbr.end(), B.nbr.begin(), B.nbr.end());
            nbr_ptr.push_back((int)nbr.size());
            halo_node.insert(halo_node.end(), B.nodes.begin(), B.nodes.end());
            halo_ptr.push_back((int)halo_node.size());
        }
        P->op_slptr.upload(slptr, s);
        P->op_blksl.upload(blksl, s);
        P->op_lcol.upload(lcol, s);
        P->op_src.upload(opsrc, s);
        {
            // the slice position of every Jacobian entry, for the set-up
            std::vector<int> opdst(P->nnz, 0);
            for (size_t e = 0; e < opsrc.size(); ++e)
                if (opsrc[e] >= 0) opdst[opsrc[e]] = (int)e;
            fd_set_op_places(c, opdst);
        }
        P->halo_ptr.upload(halo_ptr, s);
        P->halo_node.upload(halo_node, s);
        P->nbr_ptr.upload(nbr_ptr, s);
        P->nbr.upload(nbr, s);
        // the blocks' flags, then the barrier counter on its own 128-byte line
        P->flags.alloc(fused_sync_slot(nb) + 32);
        fused_reset(c);
        P->op_val.alloc(opsrc.size());
        P->op_val.zero(s);   // the padding entries stay zero
        P->op_dg.alloc(c->N);
        P->fused_nrmax = nr_max;
        P->fused_nhmax = nh_max;
        P->fused_hmax = halo_max;
        P->fused_stage = round16(P->smem_stage[1]);
        // CGS2: staged factor | row order | rows of W | direction at the
        // block's nodes; the delayed variant adds the pending vector's rows
        // and (by the cycle's length, fused_smem) the unrotated Hessenberg
        // matrix, then the block's rows of ewt and its node list; both the
        // slices' starts
        // block row arrays quad-transposed: nqp quads cover any block's rows
        // from its first quad boundary
        P->fused_nqp = nr_max / 4 + 2;
        const size_t rows = 32 * (size_t)P->fused_nqp;
        const size_t base = P->fused_stage + round16(2 * (size_t)nr_max) + rows;
        const size_t slices = 4 * ((size_t)(nr_max + 31) / 32 + 1);
        P->fused_smem = base + round16(4 * (size_t)nh_max) + slices;
        P->fused_smem_d = base + round16(4 * (size_t)nh_max) + rows + rows + 4 * (size_t)halo_max + slices;
        // one thread per row quad of the largest block, whole warps
        P->fused_threads = std::min(kFusedThreads, std::max(128, ((nr_max + 3) / 4 + 1 + 31) / 32 * 32));
        int dev = 0, coop = 0, nsm = 0;
        FVM_CUDA(cudaGetDevice(&dev));
        FVM_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
        FVM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        for (int v = 0; v < 2; ++v) {
            const void* kfn = (const void*)fused_kernel(v, P->wide);
            cudaFuncAttributes fa;
            FVM_CUDA(cudaFuncGetAttributes(&fa, kfn));
            P->fused_room[v] = kMaxDynSmem - fa.sharedSizeBytes;
            P->fused_var_ok[v] = false;
            if (fused_bytes(P, v, 1) > P->fused_room[v]) continue;
            // enough for the longest cycle, or what there is
            const size_t smem = std::min(P->fused_room[v], fused_bytes(P, v, kFusedMaxDim));
            raise_smem_limit(kfn, smem);
            // the smallest shared-memory carveout that holds the block's
            // shared data (dynamic + static, about 1 KB reserved), so that
            // the rest of the SM's 256 KB stays L1 for the block's basis rows
            const double need = (double)(smem + fa.sharedSizeBytes + 1024);
            const int pct = std::min(100, (int)std::ceil(100.0 * need / (228.0 * 1024.0)));
            FVM_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributePreferredSharedMemoryCarveout, pct));
            int per_sm = 0;
            FVM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, P->fused_threads, smem));
            P->fused_var_ok[v] = coop && per_sm > 0 && nb <= per_sm * nsm;
        }
        P->fused_ok = P->fused_var_ok[0] || P->fused_var_ok[1];
    }
    const int var = fused_variant(c);
    if (!P->fused_ok || !P->fused_var_ok[var] || fused_bytes(P, var, m) > P->fused_room[var]) return false;
    if (P->op_setup_id != P->setup_id) {
        // the values come from the set-up's kernels once the layout exists;
        // the first set-up after the layout was built copies them here
        const long nt = std::max((long)P->op_val.n, (long)c->N);
        fvm_launch(c, k_op_refresh, grid_for(nt, 256), 256, 0, s, (long)P->op_val.n, P->op_src.p, P->J.p, P->op_val.p,
                   c->N, P->lu_row.p, P->ahhp.p, c->ntype.p, P->op_dg.p);
        P->op_setup_id = P->setup_id;
    }
    return true;
}

// one cycle of at most m steps (the dimension that fused_prepare was asked for; the
// workspace K may be a larger one's) from U_0 and its squared norm (K->res[0]);
// runs until convergence, a full basis or a breakdown, and leaves the state and
// the coefficients
void fused_cycle(fvm_ctx* c, Krylov* K, int m, double cj, double tol, const double* ewt, double* H_d, double* coef) {
    BlockILU* P = c->ilu;
    cudaStream_t s = c->stream;
    float* U = reinterpret_cast<float*>(K->U);
    if (K->tdir.n < (size_t)c->N) K->tdir.alloc(c->N);
    FusedArgs a;
    a.N = c->N;
    a.m = m;
    a.nr_max = P->fused_nrmax;
    a.nqp = P->fused_nqp;
    a.nh_max = P->fused_nhmax;
    a.halo_max = P->fused_hmax;
    a.stage_max = P->fused_stage;
    a.st = K->st.p;
    a.tol = tol;
    a.sqrtN = std::sqrt((double)c->N);
    a.coef = coef;
    a.U = U;
    a.ld = K->ld;
    a.scale = K->scale.p;
    a.tdir = K->tdir.p;
    a.ewt = ewt;
    a.slptr = P->op_slptr.p;
    a.blksl = P->op_blksl.p;
    a.op_lcol = P->op_lcol.p;
    a.halo_ptr = P->halo_ptr.p;
    a.halo_node = P->halo_node.p;
    a.nbr_ptr = P->nbr_ptr.p;
    a.nbr = P->nbr.p;
    a.flags = P->flags.p;
    a.sync = P->flags.p + fused_sync_slot(P->nb);
    a.op_val = P->op_val.p;
    a.op_dg = P->op_dg.p;
    a.dcj = (float)(cj - P->cj_setup);
    a.bstart = P->bstart.p;
    a.blk = P->blk.p;
    a.lu_col = P->lu_col.p;
    a.meta = P->meta.p;
    a.lu = P->lu32.p;
    a.lu_row = P->lu_row.p;
    a.beta2 = K->res.p;
    a.partial = K->partial.p;
    a.err = K->err.p;
    a.H = H_d;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(P->nb);
    cfg.blockDim = dim3(P->fused_threads);
    const int var = fused_variant(c);
    cfg.dynamicSmemBytes = fused_bytes(P, var, m);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    // a launch takes at most 64 flag values (the last one published is m + 1) and
    // 128 barriers (CGS2: two per step); the counter has to stay below kSyncFail
    static_assert(kFusedMaxDim + 1 < 64, "flag values and barriers of a launch");
    if (P->fused_launches >= kSyncFail / (128u * (unsigned)P->nb)) fused_reset(c);
    a.base = 64u * P->fused_launches++;
    c->tm.begin(TM_CGS, s);
    FVM_CUDA(cudaLaunchKernelEx(&cfg, fused_kernel(var, P->wide), a));
    c->tm.end(TM_CGS, s);
    c->launches++;
}

} // namespace fvmb
