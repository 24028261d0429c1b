// Preconditioner: coloured finite-difference Jacobian + block-ILU(0).
//
// Set-up follows Preconditioner::setup (examples/fvmporMinlin/
// preconditioner_dss.cpp:284-373): the node-graph pattern of
// column_pattern (:107-142), the greedy distance-2 colouring of
// sequential_vertex_colouring (:61-94, neighbourhoods from
// dependent_columns :36-59), the shift
//   d_j = sqrt(eps) * max(|y_j|, |h y'_j|, 1 / w_j)          (:322-329)
// and one perturbed residual per colour (y + d on the colour's columns,
// y' + cj d) to fill J = dF/dy + cj dF/dy' column group by column group.
// The reference stores (F0 - F_shift)/d = -J; here the values are
// (F_shift - F0)/d = +J.  GMRES with a right preconditioner is unaffected
// by the sign of P, which the tests check.
//
// The reference factors that matrix with MKL DSS on the host (:368) and
// solves on the host with two PCIe copies per apply (:375-405).  Here it is
// factored on the device with ILU(0) restricted to diagonal blocks of
// contiguous node ranges (block Jacobi ILU(0), the local B_i factor of
// decomp/schur.c:887-987 without the interface Schur system).  The
// factorisation is the row-wise IKJ ILU(0) of decomp/ILU.c:12-115 with the
// pivot of row i inverted after row i is eliminated (the block branch,
// :105-107; the scalar branch at :65 indexes the pivot by the last column
// k instead of i, which is an upstream slip and not reproduced).  One CTA
// owns one block; rows are processed by dependency levels (rows of one
// level only depend on rows of earlier levels), with a barrier between
// levels, for both the factorisation and the triangular solves
// (decomp/ILU.c:133-223).
#include "cgs.cuh"
#include "ctx.cuh"
#include "ilu.cuh"
#include "krylov.cuh"
#include "tc05.cuh"

#include <algorithm>
#include <type_traits>
#include <cfloat>
#include <cmath>

namespace fvmb {

// ------------------------------------------------------------------ kernels
// ---- finite-difference Jacobian, one element at a time
// Column j of the reference's coloured difference quotient is
// (F(y + d_j e_j, y' + cj d_j e_j) - F(y, y')) / d_j (preconditioner_dss.cpp:
// 284-373): the distance-2 colouring makes every row see at most one
// perturbed node per colour, so the coloured evaluation equals these
// single-column quotients.  With the upwind directions frozen, perturbing
// node m changes only the elements that contain m, and only through h_m and
// krw(h_m): each element forms the change of its corner partials for each of
// its nodes in turn, divided by d_m,
//   dflux_f / d_m = q_f rho0 (krw'_f - krw_f) / d_m + C_fm rho0 krw'_f,
// which is the same quotient written without the cancellation of two full
// residuals.  The elements are taken kFdChunk consecutive ones per block: the
// changes stay in the block's shared memory, every non-zero (i, j) that the
// chunk touches sums its own there in ascending element order, and only that
// sum leaves the block -- the finished entry when no other chunk touches the
// non-zero, else a partial that a second kernel adds in ascending chunk order.

// per node, in one pass: the shift d = eps max(|y|, |h y'|, 1 / w); for every
// zone touching the node g = rho0 krw(h), its change dg = rho0 krw(h + d) - g
// and the quotient dg / d; what the row's diagonal subtracts (the quotient of
// the storage term y' ahh(h); on Dirichlet rows minus that of h_D - h), and the
// storage term's cj coefficient, also in FP32 at the node's place in the
// fused cycle's factor order (op_dg, once that layout exists)
struct FdNode {
    double *g, *dg, *q;        // [nz][N]
    double* diag;              // [N]
    double* ahhp;              // [N]
    float* op_dg;
    const int* lu_pos;
};
__global__ void k_fd_node(int N, const double* __restrict__ y, const double* __restrict__ yp,
                          const double* __restrict__ ewt, double hstep, double eps, double cj,
                          const ZoneDev* __restrict__ zones, int nz, const int* __restrict__ nz_ptr,
                          const int* __restrict__ nz_zone, const double* __restrict__ nz_w, double rho0,
                          const unsigned char* __restrict__ ntype, const double* __restrict__ hD, FdNode o) {
    pdl_wait_and_trigger();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const double h = y[i], ypi = yp[i];
    const double d = eps * fmax(fabs(h), fmax(fabs(hstep * ypi), 1.0 / ewt[i]));
    const double hp = h + d, rd = 1.0 / d;
    double phi = 0.0, dsw = 0.0, dswp = 0.0;
    const int p0 = nz == 1 ? i : nz_ptr[i], p1 = nz == 1 ? i + 1 : nz_ptr[i + 1];
    for (int p = p0; p < p1; ++p) {
        const int z = nz == 1 ? 0 : nz_zone[p];
        const double w = nz_w[p];
        double Sw, ds, k, dsp, kp;
        van_genuchten(h, zones[z], Sw, ds, k);
        van_genuchten(hp, zones[z], Sw, dsp, kp);
        const double dg = rho0 * (kp - k);
        o.g[(size_t)z * N + i] = rho0 * k;
        o.dg[(size_t)z * N + i] = dg;
        o.q[(size_t)z * N + i] = dg * rd;
        phi += zones[z].phi * w;
        dsw += ds * w;
        dswp += dsp * w;
    }
    const double ahh = (phi * dsw) * rho0, ahhp = (phi * dswp) * rho0;
    const bool fixed = ntype[i] != 0;
    o.diag[i] = fixed ? -(((hD[i] - hp) - (hD[i] - h)) / d) : ((ypi + cj * d) * ahhp - ypi * ahh) / d;
    o.ahhp[i] = ahhp;
    if (o.op_dg) o.op_dg[o.lu_pos[i]] = fixed ? 0.f : (float)ahhp;
}

// y = J x for the assembled difference-quotient Jacobian of the last
// set-up, shifted to another cj: the cj term of J enters only the diagonal
// of free rows, as -cj ahh(h + d) (the quotient of the storage term
// y' ahh(h), k_fd_node), so J(cj) = J(cj_setup) - (cj - cj_setup) ahh(h + d)
// on those rows.  Four lanes per row, rows in node order.
__global__ void k_jac_apply(int N, const int* __restrict__ rowptr, const int* __restrict__ col,
                            const double* __restrict__ J, const double* __restrict__ ahhp,
                            const unsigned char* __restrict__ ntype, double dcj, const double* __restrict__ x,
                            double* __restrict__ y, const int* __restrict__ skip,
                            const double* __restrict__ dcj_dev) {
    pdl_wait_and_trigger();
    if (skip && *skip) return;
    if (dcj_dev) dcj = *dcj_dev;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = g >> 2, lane = g & 3;
    if (i >= N) return;
    const int p0 = rowptr[i], p1 = rowptr[i + 1];
    double acc = 0.0;
    for (int p = p0 + lane; p < p1; p += 4) acc += J[p] * x[col[p]];
    acc += __shfl_xor_sync(0xffffffffu, acc, 1);
    acc += __shfl_xor_sync(0xffffffffu, acc, 2);
    if (lane == 0) y[i] = ntype[i] ? acc : acc - dcj * ahhp[i] * x[i];
}

// Jacobian entry q = (i, j) from its summed quotients: times 1/V_i (0 on
// Dirichlet rows), minus the row's subtrahend on the diagonal.  Written to
// the CSR values, to the place where the factorisation reads it (its block's
// copy window, contiguous, in the factor's precision) and, once the fused
// cycle's operator layout exists, to that layout.
struct FdOut {
    const double* scale;
    const double* diag;
    double* J;
    void* Jw;
    float* op_val;
    // t: the entry's places in J, Jw (-1: another block's) and op_val
    template <class S>
    __device__ __forceinline__ void store(const int4& t, double s, double scale_i, bool on_diag, double diag_i) const {
        double v = scale_i != 0.0 ? s * scale_i : 0.0;
        if (on_diag) v = v - diag_i;
        J[t.x] = v;
        if (t.y >= 0) reinterpret_cast<S*>(Jw)[t.y] = (S)v;
        if (op_val) op_val[t.z] = (float)v;
    }
};

struct FdArgs {
    int T, N, kiso, estride, nnmax;
    const int* cnode_ptr;          // [chunks + 1] nodes of each chunk
    const int* cnode;              // global ids
    const ushort4* cloc;           // [T] chunk-local corner ids
    const int2* list_at;           // [chunks] the chunk's list: first 16-byte unit, groups of 32 non-zeros
    const uint4* list;             // group offsets | places of the lanes' sums | entry-major slots
    const int* done_ptr;           // [chunks + 1] non-zeros that no other chunk touches
    const int4* done;              // place in J, Jw, op_val; 2 * chunk-local row + 1 on the diagonal
    const int* share_ptr;          // [chunks + 1] the other ones
    const int* share;              // place of the partial
    int list_max, grp_max;         // largest chunk: list words, groups
    double* part;
    const double* coef;
    const double* xyz;
    const double* eK;
    const int* ezone;
    const double* y;
    const double* g;               // [nz][N] rho0 krw, its change and quotient (k_fd_node)
    const double* dg;
    const double* gq;
    const unsigned char* upw;
    FdOut out;
};

constexpr int kFdThreads = 192;
constexpr int kFdChunk = kFdThreads;   // elements per block, one per thread
constexpr int kFdPre = 4;         // partials' places a thread fetches ahead

// shared memory of k_fd_chunk: the quotients and a zero slot; the chunk's
// nodes' h (and krw terms with one zone, coordinates when rebuilt), whose
// place the non-zeros' sums take afterwards; their rows' scale and diagonal;
// the list; its mbarrier
struct FdSmem {
    size_t nodes, rows, list, bar, bytes;
    __host__ __device__ FdSmem(int npe, bool rc, bool mz, size_t sz, int nnmax, int list_max, int grp_max) {
        const size_t nn = (size_t)nnmax * 8 * (1 + (mz ? 0 : 3) + (rc ? 3 : 0)), sums = (size_t)grp_max * 32 * 8;
        nodes = round16(((size_t)npe * npe * kFdChunk + 1) * sz);
        rows = nodes + round16(nn > sums ? nn : sums);
        list = rows + 16 * (size_t)nnmax;
        bar = list + (size_t)list_max * 2;
        bytes = bar + 16;
    }
};
// 16-bit words before the slots of a list of ng groups: ng + 1 group offsets
// (in units of 32 slots), then 32 places per group
__host__ __device__ inline int fd_list_offs(int ng) { return (ng + 8) & ~7; }

// Quotient Jacobian of one chunk of elements.  Written one by one to their
// slots in global memory, the npe^2 quotients of an element hit npe^2
// scattered sectors, and a second kernel read them back: 129 + 63 us per set-up
// on the 214k-node box (19.4 M FP32 quotients, one B200).  Here they stay in
// shared memory (column-major over the chunk's elements, so a warp writes
// consecutive words) and about two chunk sums per non-zero leave the block:
// 88 us, and 33 us for the sums over chunks (ncu, cold caches).  A block's phases
// (its nodes, its quotients, its sums, its entries) each wait on memory or on
// FP64 chains, so what counts is how many blocks share an SM: 192 elements, one
// per thread, four blocks per SM at 80 registers; 512 elements over 256 threads at two per
// SM took 108 us, 256 over 256 at three 91 us, 128 over 128 at six 92 us.
// Everything a block reads after its quotients (the list of slots, by a bulk
// copy; the sums' places) is on its way while they are formed.  The sums are
// taken longest first, a non-zero per lane, so that a warp's lanes have like
// lengths, and leave in ascending order of the non-zeros.
// Quotients are FP64, or FP32 when the factor is FP32 (which rounds every
// entry to FP32 anyway); all sums are FP64.
template <int NPE, int NFE, bool RC, bool MZ, class S>
__global__ void __launch_bounds__(kFdThreads, 4) k_fd_chunk(FdArgs a) {
    unsigned char* const smem_raw = ilu_smem();
    const FdSmem L(NPE, RC, MZ, sizeof(S), a.nnmax, a.list_max, a.grp_max);
    S* slots = reinterpret_cast<S*>(smem_raw);
    double* sh = reinterpret_cast<double*>(smem_raw + L.nodes);
    double* sg = sh + a.nnmax;                  // one zone: g, dg, quotient
    double* sx = sh + (MZ ? 1 : 4) * a.nnmax;   // rebuilt geometry
    double* sums = sh;
    double2* srow = reinterpret_cast<double2*>(smem_raw + L.rows);
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem_raw + L.bar);
    pdl_wait_and_trigger();
    const int2 la = a.list_at[blockIdx.x];
    const int ng = la.y;
    const unsigned short* goff = reinterpret_cast<const unsigned short*>(smem_raw + L.list);
    const unsigned short* lrank = goff + fd_list_offs(ng);
    const unsigned short* lslot = lrank + 32 * ng;
    if (threadIdx.x == 0) {
        tc05::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        const uint32_t bytes = 16u * (uint32_t)(a.list_at[blockIdx.x + 1].x - la.x);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc05::smem_u32(bar)), "r"(bytes)
                     : "memory");
        tc05::bulk_g2s(smem_raw + L.list, a.list + la.x, bytes, bar);
    }
    const int e0 = blockIdx.x * kFdChunk, ne = min(kFdChunk, a.T - e0);
    const int el = threadIdx.x, e = e0 + el;
    // the element's record
    ushort4 lq = make_ushort4(0, 0, 0, 0);
    uint2 uc = make_uint2(0u, 0u);
    double K0 = 0.0, K1 = 0.0, K2 = 0.0;
    if (el < ne) {
        lq = a.cloc[e];
        uc = *reinterpret_cast<const uint2*>(a.upw + (size_t)8 * e);
        if (RC) {
            K0 = K1 = K2 = a.eK[e];
            if (!a.kiso) {
                K1 = a.eK[(size_t)a.estride + e];
                K2 = a.eK[(size_t)2 * a.estride + e];
            }
        }
    }
    const int n0 = a.cnode_ptr[blockIdx.x], nn = a.cnode_ptr[blockIdx.x + 1] - n0;
    for (int k = threadIdx.x; k < nn; k += kFdThreads) {
        const int g = a.cnode[n0 + k];
        sh[k] = a.y[g];
        srow[k] = make_double2(a.out.scale[g], a.out.diag[g]);
        if (!MZ) {
            sg[k] = a.g[g];
            sg[a.nnmax + k] = a.dg[g];
            sg[2 * a.nnmax + k] = a.gq[g];
        }
        if (RC) {
            sx[k] = a.xyz[g];
            sx[a.nnmax + k] = a.xyz[(size_t)a.N + g];
            sx[2 * a.nnmax + k] = a.xyz[(size_t)2 * a.N + g];
        }
    }
    if (threadIdx.x == 0) slots[NPE * NPE * kFdChunk] = (S)0;
    __syncthreads();
    if (el < ne) {
        const int li[4] = {lq.x, lq.y, lq.z, lq.w};
        double gk[NPE], dg[NPE], gq[NPE];
        if (MZ) {
            const size_t zo = (size_t)a.ezone[e] * a.N;
#pragma unroll
            for (int k = 0; k < NPE; ++k) {
                const size_t g = zo + a.cnode[n0 + li[k]];
                gk[k] = a.g[g];
                dg[k] = a.dg[g];
                gq[k] = a.gq[g];
            }
        } else {
#pragma unroll
            for (int k = 0; k < NPE; ++k) {
                gk[k] = sg[li[k]];
                dg[k] = sg[a.nnmax + li[k]];
                gq[k] = sg[2 * a.nnmax + li[k]];
            }
        }
        // C[f][m] of column m: with the rebuilt geometry the face
        // combinations of one column of the cofactor rows' Gram matrix
        double q[NFE];
        TetGram G;
        if constexpr (RC) {
            double X[4][3];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                X[k][0] = sx[li[k]];
                X[k][1] = sx[a.nnmax + li[k]];
                X[k][2] = sx[2 * a.nnmax + li[k]];
            }
            G = tet_gram(X[0], X[1], X[2], X[3], K0, K1, K2);
            G.fluxes(sh[li[0]], sh[li[1]], sh[li[2]], sh[li[3 % NPE]], q);
        } else {
#pragma unroll
            for (int f = 0; f < NFE; ++f) {
                const double* cf = a.coef + (size_t)(f * (NPE + 1)) * a.T + e;
                double s = cf[0] * sh[li[0]];
#pragma unroll
                for (int k = 1; k < NPE; ++k) s += cf[(size_t)k * a.T] * sh[li[k]];
                q[f] = s + cf[(size_t)NPE * a.T];
            }
        }
        // upwind weights of each face's ends (1 and 0, or halves before the
        // first step), the face's rho0 krw, and what its ends' own columns add
        // to C rho0 krw: q times the quotient, C times the change
        double gf[NFE], wa[NFE];
#pragma unroll
        for (int f = 0; f < NFE; ++f) {
            const int fa = NPE == 4 ? tet_edge_a(f) : tri_edge_a(f);
            const int fb = NPE == 4 ? tet_edge_b(f) : tri_edge_b(f);
            const unsigned u = (f < 4 ? uc.x >> (8 * f) : uc.y >> (8 * (f - 4))) & 0xffu;
            wa[f] = u == 0 ? 1.0 : (u == 1 ? 0.0 : 0.5);
            gf[f] = wa[f] * gk[fa] + (1.0 - wa[f]) * gk[fb];
        }
#pragma unroll
        for (int m = 0; m < NPE; ++m) {
            double C[NFE], dc[NPE];
            if constexpr (RC) {
                G.column(m, C);
            } else {
#pragma unroll
                for (int f = 0; f < NFE; ++f) C[f] = a.coef[(size_t)(f * (NPE + 1) + m) * a.T + e];
            }
#pragma unroll
            for (int k = 0; k < NPE; ++k) dc[k] = 0.0;
#pragma unroll
            for (int f = 0; f < NFE; ++f) {
                const int fa = NPE == 4 ? tet_edge_a(f) : tri_edge_a(f);
                const int fb = NPE == 4 ? tet_edge_b(f) : tri_edge_b(f);
                double df = C[f] * gf[f];
                if (fa == m || fb == m) df += (fa == m ? wa[f] : 1.0 - wa[f]) * (q[f] * gq[m] + C[f] * dg[m]);
                dc[fa] -= df;
                dc[fb] += df;
            }
#pragma unroll
            for (int k = 0; k < NPE; ++k) slots[(m * NPE + k) * kFdChunk + el] = (S)dc[k];
        }
    }
    const int d0 = a.done_ptr[blockIdx.x], nd = a.done_ptr[blockIdx.x + 1] - d0;
    const int s0 = a.share_ptr[blockIdx.x], ns = a.share_ptr[blockIdx.x + 1] - s0;
    // the sums' places, on their way while the sums are taken
    int shr[kFdPre];
#pragma unroll
    for (int k = 0; k < kFdPre; ++k) {
        const int p = threadIdx.x + k * kFdThreads;
        shr[k] = p < ns ? a.share[s0 + p] : 0;
    }
    const int4 first = (int)threadIdx.x < nd ? a.done[d0 + threadIdx.x] : make_int4(0, -1, 0, 0);
    // the list has landed; a block that gave up waiting for it would read
    // unfilled shared memory, so it leaves its entries NaN (the solve fails)
    const bool ok = tc05::mbar_wait(bar, 0) || tc05::mbar_wait(bar, 0);
    const bool good = __syncthreads_and(ok ? 1 : 0) != 0;
    // a warp's lanes each sum one non-zero; the lanes of a group are padded
    // to its longest with the zero slot
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (good) {
        for (int g = warp; g < ng; g += kFdThreads / 32) {
            const int o1 = 32 * goff[g + 1];
            double s = 0.0;
#pragma unroll 4
            for (int o = 32 * goff[g] + lane; o < o1; o += 32) s += (double)slots[lslot[o]];
            sums[lrank[32 * g + lane]] = s;
        }
    } else {
        for (int p = threadIdx.x; p < nd + ns; p += kFdThreads) sums[p] = nan("");
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kFdPre; ++k) {
        const int p = threadIdx.x + k * kFdThreads;
        if (p < ns) a.part[shr[k]] = sums[nd + p];
    }
    for (int p = threadIdx.x + kFdPre * kFdThreads; p < ns; p += kFdThreads) a.part[a.share[s0 + p]] = sums[nd + p];
    for (int p = threadIdx.x; p < nd; p += kFdThreads) {
        const int4 t = p < kFdThreads ? first : a.done[d0 + p];
        const double2 r = srow[t.w >> 1];
        a.out.store<S>(t, sums[p], r.x, t.w & 1, r.y);
    }
}

// the non-zeros touched by several chunks: their partials in ascending
// chunk order.  at: place in J, Jw and op_val, and 2 * row + 1 on the diagonal
template <class S>
__global__ void k_fd_shared(int n, const int4* __restrict__ at, const int* __restrict__ sptr,
                            const double* __restrict__ part, FdOut out) {
    pdl_wait_and_trigger();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int4 w = at[t];
    const int p0 = sptr[t], p1 = sptr[t + 1];
    const double scale = out.scale[w.w >> 1], diag = w.w & 1 ? out.diag[w.w >> 1] : 0.0;
    double s = 0.0;
    for (int p = p0; p < p1; ++p) s += part[p];
    out.store<S>(w, s, scale, w.w & 1, diag);
}

// Factorisation and sweeps of a block whose window does not fit into shared
// memory, in place in global memory.  Row i's entries in column order: its
// lower ones, the pivot, its upper ones (up[] gives an upper lane's place).  A row
// per thread, whose chain of dependent loads is what it waits for: levels of a few
// hundred rows want as many threads.
constexpr int kIluPlainFactorThreads = 512;
template <class T>
__global__ void __launch_bounds__(kIluPlainFactorThreads, 1) k_ilu_factor(const int* __restrict__ bstart, const IluBlk* __restrict__ blk,
                                                    const unsigned short* __restrict__ meta, const int* __restrict__ up,
                                                    const T* __restrict__ Jw,
                                                    const unsigned short* __restrict__ lu_col, T* lu, int* status) {
    const IluBlk B = blk[blockIdx.x];
    const int r0 = bstart[blockIdx.x], nr = bstart[blockIdx.x + 1] - r0;
    const long wn = (long)ilu_window(nr, B.ds);
    T* val = lu + B.v0;
    for (long p = threadIdx.x; p < wn; p += blockDim.x) val[p] = Jw[B.v0 + p];
    __syncthreads();
    const auto V = ilu_in_place<T>(B, nr, lu, lu_col, meta);
    const int D = B.ds;
    for (int l = 0; l < B.nl; ++l) {
        const int q1 = kIluGroup * ilu_level(V, false, l + 1);
        for (int q = kIluGroup * ilu_level(V, false, l) + threadIdx.x; q < q1; q += blockDim.x) {
            const int i = ilu_row(V, false, q / kIluGroup, q % kIluGroup);
            if (i == kIluNoRow) continue;
            const IluSpan lo = ilu_span(V, false, q / kIluGroup, q % kIluGroup);
            const int ui = up[r0 + i];
            const IluSpan hi = ilu_span(V, true, ui / kIluGroup, ui % kIluGroup);
            for (int kk = 0; kk < lo.w; ++kk) {
                const int p = lo.entry(kk), k = (int)V.col(p);
                if (k == nr) break;
                const T lik = val[p] * val[D + k];
                val[p] = lik;
                // U(k) against the rest of row i
                const int uk = up[r0 + k];
                const IluSpan ku = ilu_span(V, true, uk / kIluGroup, uk % kIluGroup);
                int a = kk + 1, c = 0;
                for (int u = 0; u < ku.w; ++u) {
                    const int j = (int)V.col(ku.entry(u));
                    if (j == nr) break;
                    int at = -1;
                    if (j < i) {
                        while (a < lo.w && (int)V.col(lo.entry(a)) < j) ++a;
                        if (a < lo.w && (int)V.col(lo.entry(a)) == j) at = lo.entry(a);
                    } else if (j == i) {
                        at = D + i;
                    } else {
                        while (c < hi.w && (int)V.col(hi.entry(c)) < j) ++c;
                        if (c < hi.w && (int)V.col(hi.entry(c)) == j) at = hi.entry(c);
                    }
                    if (at >= 0) val[at] = val[at] - lik * val[ku.entry(u)];
                }
            }
            T d = val[D + i];
            if (d == (T)0 || !isfinite((double)d)) {
                atomicExch(status, 1);
                d = (T)1;
            }
            val[D + i] = (T)1 / d;
        }
        __syncthreads();
    }
}

template <class T>
__global__ void __launch_bounds__(kIluThreads) k_ilu_apply(const int* __restrict__ bstart, const IluBlk* __restrict__ blk,
                                                   const unsigned short* __restrict__ lu_col,
                                                   const unsigned short* __restrict__ meta, const T* __restrict__ lu,
                                                   const int* __restrict__ lu_row, const double* __restrict__ r,
                                                   double* __restrict__ z, const int* __restrict__ skip) {
    unsigned char* const smem_raw = ilu_smem();
    pdl_wait_and_trigger();
    if (skip && *skip) return;
    T* x = reinterpret_cast<T*>(smem_raw);
    const IluBlk B = blk[blockIdx.x];
    const int r0 = bstart[blockIdx.x], nr = bstart[blockIdx.x + 1] - r0;
    for (int i = threadIdx.x; i < nr; i += blockDim.x) x[i] = (T)r[lu_row[r0 + i]];
    __syncthreads();
    const auto V = ilu_in_place(B, nr, lu, lu_col, meta);
    // level 0 of the lower sweep has no off-diagonal entries
    ilu_sweep_any<T, false>(V, 1, V.nl);
    ilu_sweep_any<T, true>(V, 0, V.nu);
    for (int i = threadIdx.x; i < nr; i += blockDim.x) z[lu_row[r0 + i]] = (double)x[i];
}

template <class T, bool WIDE>
__global__ void __launch_bounds__(kIluThreads, 1) k_ilu_apply_smem(const int* __restrict__ bstart,
                                                        const IluBlk* __restrict__ blk,
                                                        const unsigned short* __restrict__ lu_col,
                                                        const unsigned short* __restrict__ meta,
                                                        const T* __restrict__ lu,
                                                        const int* __restrict__ lu_row,
                                                        const double* __restrict__ r,
                                                        double* __restrict__ z, int* __restrict__ err,
                                                        const int* __restrict__ skip) {
    unsigned char* const smem_raw = ilu_smem();
    const IluBlk B = blk[blockIdx.x];
    const int r0 = bstart[blockIdx.x], nr = bstart[blockIdx.x + 1] - r0;
    const IluStage<T> S(B, nr);
    T* x = S.x;
    if (threadIdx.x == 0) {
        tc05::mbar_init(S.bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    __syncthreads();
    // factor window, columns and the block's record by three bulk copies; the
    // right-hand side by the threads meanwhile.  The copies read only set-up
    // data, so they are issued before the wait for the previous kernel (the
    // factorisation has completed before any kernel that lets this launch
    // start early: the copy of the status word lies between, psetup_dev); the
    // right-hand side and the skip flag are read after it.
    ilu_stage_bulk(S, B, nr, lu, lu_col, meta);
    // the nodes of the thread's rows, for the way in and the way out: set-up data
    // too, and with them at hand the right-hand side is one round of loads
    // (17.0 us per apply on the 214k-node box with both read row by row)
    constexpr int kRows = 8;
    int node[kRows];
#pragma unroll
    for (int k = 0; k < kRows; ++k) node[k] = lu_row[r0 + min((int)(threadIdx.x + k * blockDim.x), nr - 1)];
    pdl_wait_and_trigger();
    if (skip && *skip) {
        // a step queued after the stop: let the copies land (bounded), leave
        tc05::mbar_wait(S.bar, 0);
        return;
    }
    {
        double v[kRows];
#pragma unroll
        for (int k = 0; k < kRows; ++k) v[k] = threadIdx.x + k * blockDim.x < nr ? r[node[k]] : 0.0;
#pragma unroll
        for (int k = 0; k < kRows; ++k)
            if (threadIdx.x + k * blockDim.x < nr) x[threadIdx.x + k * blockDim.x] = (T)v[k];
    }
    for (int i = threadIdx.x + kRows * blockDim.x; i < nr; i += blockDim.x) x[i] = (T)r[lu_row[r0 + i]];
    if (threadIdx.x == 0) x[nr] = (T)0;
    bool ok = tc05::mbar_wait(S.bar, 0);
    if (!ok) ok = tc05::mbar_wait(S.bar, 0);   // copies in flight get a second bounded chance
    if (!__syncthreads_and(ok ? 1 : 0)) {
        // the factor never arrived: report it and pass the vector through
        // unpreconditioned instead of reading unfilled shared memory
        if (threadIdx.x == 0) atomicExch(err, 2);
        for (int i = threadIdx.x; i < nr; i += blockDim.x) z[lu_row[r0 + i]] = (double)x[i];
        return;
    }
    const IluShared<T> V = S.view(B);
    // level 0 of the lower sweep has no off-diagonal entries
    ilu_sweep<T, false, WIDE>(V, 1, V.nl);
    ilu_sweep<T, true, WIDE>(V, 0, V.nu);
#pragma unroll
    for (int k = 0; k < kRows; ++k)
        if (threadIdx.x + k * blockDim.x < nr) z[node[k]] = (double)x[threadIdx.x + k * blockDim.x];
    for (int i = threadIdx.x + kRows * blockDim.x; i < nr; i += blockDim.x) z[lu_row[r0 + i]] = (double)x[i];
}

// Block ILU(0) coupled through the Schur complement of the block
// interfaces (decomp/schur.c:1407-1636, precon_schur_apply).  Each block's
// factor is ordered [interior B; interface] so that it reads
//   [L_B 0; F~ L_S] [U_B E~; 0 U_S],
// L_S U_S being the ILU(0) of the block's local Schur complement
// C - F B^-1 E on C's pattern; the interface system of the whole matrix is
// S = L_S U_S + C_o, C_o the couplings to the other blocks' interface rows.
// One cooperative launch, one CTA per block, the factor staged in shared
// memory once for the whole apply, or read in place where its padding keeps
// that from fitting (STAGED false, schur_layout):
//   z = L^-1 r (the forward sweep; x_L = M_B f and g - F x_L of the
//     reference), kept in shared memory;
//   x_S = U_S^-1 z_S, then `iters` times: publish x_S, grid barrier,
//     x_S <- U_S^-1 (z_S - L_S^-1 C_o x_S) with the other blocks' published
//     values (block-Jacobi sweeps on S, the reference's level-0 solve);
//   x_B = U_B^-1 (z_B - E~ x_S) (x_L = M_B (f - E y)).
// The published iterates alternate between two node-order buffers, so a
// block still reading sweep i never sees sweep i + 1's values.  Barrier
// waits are bounded (error 3 in serr, every block leaves at its next
// barrier); a factor that never reached shared memory passes r through and
// records error 2, as the staged apply does.
template <class T> struct SchurArgs {
    int N, iters;
    size_t stage_max;          // offset of the forward result in shared memory
    const int* bstart;
    const IluBlk* blk;
    const unsigned short* lu_col;
    const unsigned short* meta;
    const T* lu;
    const int* lu_row;
    const int* sch_lv;
    const int* sch_nin;
    const int* o_ptr;
    const int* o_col;
    const int* o_src;
    const double* J;
    double* xg;
    unsigned* bar;
    int* serr;
    const double* r;
    double* z;
    int* err;
    const int* skip;
};

// (registers for as many CTAs of 256 threads per SM as blocks may have to be
// resident: four in FP32, three in FP64)
template <class T, bool STAGED>
__global__ void __launch_bounds__(kIluThreads, sizeof(T) == 4 ? 4 : 3) k_ilu_apply_schur(SchurArgs<T> a) {
    unsigned char* const smem_raw = ilu_smem();
    const int b = blockIdx.x;
    const IluBlk B = a.blk[b];
    const int r0 = a.bstart[b], nr = a.bstart[b + 1] - r0;
    const IluStage<T> S(B, nr);
    T* x = S.x;
    uint64_t* mbar = S.bar;
    T* zs = reinterpret_cast<T*>(smem_raw + a.stage_max);
    if constexpr (STAGED) {
        if (threadIdx.x == 0) {
            tc05::mbar_init(mbar, 1);
            asm volatile("fence.mbarrier_init.release.cluster;");
        }
        __syncthreads();
        ilu_stage_bulk(S, B, nr, a.lu, a.lu_col, a.meta);
    }
    pdl_wait_and_trigger();
    if (a.skip && *a.skip) {
        // a step queued after the stop: every block leaves before any barrier
        if constexpr (STAGED) tc05::mbar_wait(mbar, 0);
        return;
    }
    for (int i = threadIdx.x; i < nr; i += blockDim.x) x[i] = (T)a.r[a.lu_row[r0 + i]];
    if (STAGED && threadIdx.x == 0) x[nr] = (T)0;
    bool ok = true;
    if constexpr (STAGED) ok = tc05::mbar_wait(mbar, 0) || tc05::mbar_wait(mbar, 0);
    const bool good = __syncthreads_and(ok ? 1 : 0) != 0;
    if (!good && threadIdx.x == 0) atomicExch(a.err, 2);
    const int lvB = a.sch_lv[2 * b], uvS = a.sch_lv[2 * b + 1], nin = a.sch_nin[b];
    const auto V = [&] {
        if constexpr (STAGED) return S.view(B);
        else return ilu_in_place(B, nr, a.lu, a.lu_col, a.meta);
    }();
    if (good) {
        ilu_sweep_any<T, false>(V, 1, V.nl);
        for (int i = threadIdx.x; i < nr; i += blockDim.x) zs[i] = x[i];
        __syncthreads();
        ilu_sweep_any<T, true>(V, 0, uvS);
    }
    for (int it = 0; it < a.iters; ++it) {
        double* xo = a.xg + (size_t)(it & 1) * a.N;
        if (good)
            for (int q = nin + threadIdx.x; q < nr; q += blockDim.x) xo[a.lu_row[r0 + q]] = (double)x[q];
        // a block without its factor still takes part in every barrier
        if (!grid_barrier(a.bar, a.bar + 1, a.serr)) return;
        if (!good) continue;
        for (int q = threadIdx.x; q < nin; q += blockDim.x) x[q] = (T)0;
        for (int q = nin + threadIdx.x; q < nr; q += blockDim.x) {
            T acc = (T)0;
            const int e1 = a.o_ptr[r0 + q + 1];
            for (int e = a.o_ptr[r0 + q]; e < e1; ++e) acc += (T)a.J[a.o_src[e]] * (T)__ldcg(xo + a.o_col[e]);
            x[q] = acc;
        }
        __syncthreads();
        ilu_sweep_any<T, false>(V, lvB, V.nl);
        for (int q = nin + threadIdx.x; q < nr; q += blockDim.x) x[q] = zs[q] - x[q];
        __syncthreads();
        ilu_sweep_any<T, true>(V, 0, uvS);
    }
    if (!good) {
        for (int i = threadIdx.x; i < nr; i += blockDim.x) a.z[a.lu_row[r0 + i]] = (double)x[i];
        return;
    }
    if (a.iters > 0) {
        for (int q = threadIdx.x; q < nin; q += blockDim.x) x[q] = zs[q];
        __syncthreads();
    }
    ilu_sweep_any<T, true>(V, uvS, V.nu);
    for (int i = threadIdx.x; i < nr; i += blockDim.x) a.z[a.lu_row[r0 + i]] = (double)x[i];
}

static const void* schur_kernel(int precision, bool staged) {
    if (precision) return staged ? (const void*)k_ilu_apply_schur<float, true> : (const void*)k_ilu_apply_schur<float, false>;
    return staged ? (const void*)k_ilu_apply_schur<double, true> : (const void*)k_ilu_apply_schur<double, false>;
}

// Whether the coupled apply runs on these blocks, and how.  It keeps each block's
// forward result in shared memory through its grid barriers, and all blocks
// must be resident at once.  It is offered where the factor's own entries (rows
// end to end, with row pointers and level lists: `exact` bytes for the largest
// block) fit beside that.  The window that the sweeps read is padded, by up to 5 %
// on small blocks in this order; where only the padding is too much, the sweeps
// read the factor in place.
static void schur_layout(const fvm_ctx* c, BlockILU* P, int pr, size_t exact) {
    int nsm = 148, coop = 0;
    FVM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device));
    FVM_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device));
    P->schur_smem[pr] = 0;
    if (!coop) return;
    const size_t sz = pr ? sizeof(float) : sizeof(double), fwd = round16(sz * (size_t)P->maxb);
    auto resident = [&](bool staged, size_t bytes) {
        if (bytes > kMaxDynSmem) return false;
        const void* kfn = schur_kernel(pr, staged);
        raise_smem_limit(kfn, bytes);
        int per_sm = 0;
        FVM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, P->apply_threads, bytes));
        return (long)per_sm * nsm >= P->nb;
    };
    if (!exact || !resident(true, round16(exact) + fwd)) return;
    const size_t staged = round16(P->smem_stage[pr]) + fwd, plain = round16(ilu_plain_bytes(P->maxb, sz)) + fwd;
    P->schur_staged[pr] = P->smem_stage[pr] && resident(true, staged);
    if (P->schur_staged[pr]) P->schur_smem[pr] = staged;
    else if (resident(false, plain)) P->schur_smem[pr] = plain;
}

template <class T>
static void launch_schur_apply(fvm_ctx* c, BlockILU* P, const T* lu, const double* r, double* z, const int* skip) {
    SchurArgs<T> a;
    a.N = c->N;
    a.iters = P->schur_iters;
    const bool staged = P->schur_staged[P->factored];
    a.stage_max = staged ? round16(P->smem_stage[P->factored]) : round16(ilu_plain_bytes(P->maxb, sizeof(T)));
    a.bstart = P->bstart.p;
    a.blk = P->blk.p;
    a.lu_col = P->lu_col.p;
    a.meta = P->meta.p;
    a.lu = lu;
    a.lu_row = P->lu_row.p;
    a.sch_lv = P->sch_lv.p;
    a.sch_nin = P->sch_nin.p;
    a.o_ptr = P->o_ptr.p;
    a.o_col = P->o_col.p;
    a.o_src = P->o_src.p;
    a.J = P->J.p;
    a.xg = P->xg.p;
    a.bar = P->sbar.p;
    a.serr = P->serr.p;
    a.r = r;
    a.z = z;
    a.err = P->status.p;
    a.skip = skip;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(P->nb);
    cfg.blockDim = dim3(P->apply_threads);
    cfg.dynamicSmemBytes = P->schur_smem[P->factored];
    cfg.stream = c->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    if (staged) FVM_CUDA(cudaLaunchKernelEx(&cfg, k_ilu_apply_schur<T, true>, a));
    else FVM_CUDA(cudaLaunchKernelEx(&cfg, k_ilu_apply_schur<T, false>, a));
    c->launches++;
}

// Shared-memory factorisation: bring the block's Jacobian entries into the
// same copy window the apply uses, eliminate level by level in shared
// memory (IKJ, pivots inverted after their row), write the block back.
// 1024 threads: one block per SM, so the schedule prefetch and the copy out
// keep many loads in flight.  A row's updates by one L entry touch different
// entries, so four lanes share a row: the row's chain per L entry is one or
// two updates instead of up to eight, and a level's rows (a few hundred) keep
// all the warps busy.  Schedule words of the next level each thread holds:
constexpr int kIluFactorThreads = 1024;
constexpr int kIluFactorPre = 8;
constexpr int kIluFactorLanes = 4;

template <class T>
__global__ void __launch_bounds__(kIluFactorThreads, 1) k_ilu_factor_smem(const int* __restrict__ bstart,
                                                         const IluBlk* __restrict__ blk,
                                                         const unsigned short* __restrict__ meta,
                                                         const T* __restrict__ Jw,
                                                         const unsigned short* __restrict__ lu_col,
                                                         const int* __restrict__ seg_ptr,
                                                         const unsigned* __restrict__ upd, int scr_off,
                                                         int scr_words, T* __restrict__ lu,
                                                         int* status) {
    unsigned char* const smem_raw = ilu_smem();
    const int b = blockIdx.x;
    const IluBlk B = blk[b];
    const int r0 = bstart[b], nr = bstart[b + 1] - r0;
    const IluStage<T> S(B, nr);
    T* const val = S.val;
    if (threadIdx.x == 0) {
        tc05::mbar_init(S.bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    __syncthreads();
    pdl_wait_and_trigger();
    ilu_stage_bulk(S, B, nr, Jw, lu_col, meta);
    const int la = B.seg, nl = B.nl;
    // Each level's schedule segment is in shared memory when its rows run
    // (read in place from global when it is larger than a buffer), so a
    // row's update chain never waits on global loads: two buffers; while a
    // level's rows run, every thread holds its share of the next level's
    // segment in registers (loads issued before the rows, stored after).
    unsigned* const buf0 = reinterpret_cast<unsigned*>(smem_raw + scr_off);
    unsigned* const buf1 = buf0 + scr_words;
    int sgc = seg_ptr[la], lenc = seg_ptr[la + 1] - sgc;
    bool cur_smem = lenc <= scr_words;
    if (cur_smem) {
#pragma unroll 4
        for (int t = threadIdx.x; t < lenc; t += blockDim.x) buf0[t] = upd[sgc + t];
    }
    bool ok = tc05::mbar_wait(S.bar, 0);
    if (!ok) ok = tc05::mbar_wait(S.bar, 0);   // copies in flight get a second bounded chance
    if (!__syncthreads_and(ok ? 1 : 0)) {
        // the block never arrived: report it as a failed factorisation
        if (threadIdx.x == 0) atomicExch(status, 2);
        return;
    }
    const IluShared<T> V = S.view(B);
    const int D = B.ds;
    constexpr int G = kIluFactorLanes, R = 32 / (G * kIluGroup);   // lanes per row, groups per warp
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int l = 0; l < nl; ++l) {
        int sgn = 0, lenn = 0;
        bool nxt_smem = false;
        unsigned pre[kIluFactorPre];
        if (l + 1 < nl) {
            sgn = seg_ptr[la + l + 1];
            lenn = seg_ptr[la + l + 2] - sgn;
            nxt_smem = lenn <= scr_words;
            if (nxt_smem) {
#pragma unroll
                for (int i = 0; i < kIluFactorPre; ++i) {
                    const int t = threadIdx.x + i * blockDim.x;
                    pre[i] = t < lenn ? upd[sgn + t] : 0u;
                }
            }
        }
        const unsigned* L = cur_smem ? ((l & 1) ? buf1 : buf0) : upd + sgc;
        const int g0 = ilu_level(V, false, l), g1 = ilu_level(V, false, l + 1);
        // a warp takes R consecutive groups; the first has the longest rows
        for (int gw = g0 + R * warp; gw < g1; gw += R * nw) {
            const int gr = gw + lane / (G * kIluGroup), q = lane / G % kIluGroup, g = lane % G;
            const int i = gr < g1 ? ilu_row(V, false, gr, q) : kIluNoRow;
            const IluSpan S = ilu_span(V, false, min(gr, g1 - 1), q);
            const int w = __shfl_sync(0xffffffffu, S.w, 0);
            const bool row = i != kIluNoRow;
            // IKJ with the precomputed schedule: the updates of each L entry,
            // in the order a merge of the row with U(k) would find them
            int t = row ? (int)L[kIluGroup * (gr - g0) + q] : 0;
            for (int kk = 0; kk < w; ++kk) {
                const bool in = row && kk < S.w;
                const int p = S.entry(in ? kk : 0);
                const int k = in ? (int)V.col(p) : nr;
                const bool act = k != nr;
                T lik = (T)0;
                if (act) {
                    const int cnt = (int)L[t];
                    lik = val[p] * val[D + k];
                    for (int u = g; u < cnt; u += G) {
                        const unsigned pr = L[t + 1 + u];
                        const int jj = (int)(pr & 0xffffu), kp = (int)(pr >> 16);
                        val[jj] = val[jj] - lik * val[kp];
                    }
                    t += 1 + cnt;
                }
                __syncwarp();
                // the entry itself was read by the row's other lanes above
                if (act && g == 0) val[p] = lik;
            }
            if (row && g == 0) {
                T d = val[D + i];
                if (d == (T)0 || !isfinite((double)d)) {
                    atomicExch(status, 1);
                    d = (T)1;
                }
                val[D + i] = (T)1 / d;
            }
        }
        if (nxt_smem) {
            unsigned* nb = (l & 1) ? buf0 : buf1;   // the buffer of level l - 1, finished
#pragma unroll
            for (int i = 0; i < kIluFactorPre; ++i) {
                const int t = threadIdx.x + i * blockDim.x;
                if (t < lenn) nb[t] = pre[i];
            }
        }
        __syncthreads();
        sgc = sgn;
        lenc = lenn;
        cur_smem = nxt_smem;
    }
    const int wn = (int)ilu_window(nr, B.ds);
    for (int p = threadIdx.x; p < wn; p += blockDim.x) lu[B.v0 + p] = val[p];
}

// ------------------------------------------------------------------ host set-up
// Colour order of the rows [r0, r1) of a block (offsets from r0): greedy
// colouring in natural order over the couplings inside the block, then
// stable by colour.  The CPU oracle restates the same rule.
//
// With interface_last (Schur coupling) the rows coupled to a node outside the
// block (interface rows) follow all interior rows: the sort key is
// (interface, colour); *n_interior gets the number of interior rows.
static std::vector<int> block_colour_order(const std::vector<int>& rp, const std::vector<int>& cl, int r0, int r1,
                                           bool interface_last = false, int* n_interior = nullptr) {
    const int nr = r1 - r0;
    std::vector<int> colour(nr, 0), ord(nr), key(nr);
    int ncol = 1, nin = 0;
    for (int i = r0; i < r1; ++i) {
        unsigned long long used = 0ull;
        std::vector<int> more;
        bool iface = false;
        for (int p = rp[i]; p < rp[i + 1]; ++p) {
            const int j = cl[p];
            if (j < r0 || j >= r1) iface = true;
            if (j < r0 || j >= i) continue;
            const int cj = colour[j - r0];
            if (cj < 64) used |= 1ull << cj;
            else more.push_back(cj);
        }
        int cc = 0;
        while (cc < 64 && ((used >> cc) & 1ull)) ++cc;
        if (cc == 64) {
            std::sort(more.begin(), more.end());
            for (int m : more)
                if (m == cc) ++cc;
        }
        colour[i - r0] = cc;
        key[i - r0] = interface_last && iface ? (1 << 20) + cc : cc;
        if (!iface) ++nin;
        ncol = std::max(ncol, cc + 1);
    }
    if (n_interior) *n_interior = interface_last ? nin : nr;
    for (int ii = 0; ii < nr; ++ii) ord[ii] = ii;
    std::stable_sort(ord.begin(), ord.end(), [&](int a, int b2) { return key[a] < key[b2]; });
    return ord;
}

// Tables of the quotient Jacobian's chunks (k_fd_chunk): the distinct nodes of
// every chunk with the elements' local corner ids; the non-zeros it touches,
// first those no other chunk touches, then the others with the places of
// their partials, each ascending; and the list of all of them longest first
// in groups of 32, with their slots in ascending element order.  The places
// in the operator layout (done, shared: .z) follow once that layout exists.
struct FdTables {
    std::vector<int> cnode_ptr, cnode, done_ptr, share_ptr, share, sptr;
    std::vector<int2> list_at;
    std::vector<int4> done, shared;
    std::vector<ushort4> cloc;
    std::vector<unsigned short> list;
    int nnmax = 0, list_max = 0, grp_max = 0;
};

// greedy distance-2 colouring in node order (preconditioner_dss.cpp:61-94): the
// number of residuals the reference's set-up takes.  The element-wise quotients
// do not use it, so it is formed when asked for (fvm_precond_info).
static int count_colours(const std::vector<int>& rp, const std::vector<int>& cl) {
    const int N = (int)rp.size() - 1;
    std::vector<int> colour(N, -1), cmark(N + 1, -1);
    int maxc = 0;
    for (int i = 0; i < N; ++i) {
        for (int p = rp[i]; p < rp[i + 1]; ++p) {
            const int nb = cl[p];
            for (int q = rp[nb]; q < rp[nb + 1]; ++q) {
                const int cc = colour[cl[q]];
                if (cc >= 0) cmark[cc] = i;
            }
        }
        int cc = 0;
        while (cc < maxc && cmark[cc] == i) ++cc;
        if (cc == maxc) ++maxc;
        colour[i] = cc;
    }
    return maxc;
}

static void build_fd_tables(const fvm_ctx* c, const BlockILU* P, const std::vector<int>& rowof,
                            const std::vector<int>& lu_dst, FdTables& fd) {
    const int T = c->T, npe = c->npe, npe2 = npe * npe;
    const std::vector<int>&rp = P->h_rowptr, &cl = P->h_col;
    const int nch = (T + kFdChunk - 1) / kFdChunk;
    // every chunk by itself: its nodes, its non-zeros (qs) and the slots of each
    // (cnt many from pos on, ascending element)
    struct Chunk {
        std::vector<int> nodes, qs, cnt, pos;
        std::vector<unsigned short> slots;
        // then, once it is known which other chunks touch them
        std::vector<int4> done;
        std::vector<int> shared;
        std::vector<unsigned short> list;
        int ng = 0;
    };
    std::vector<Chunk> chunk(nch);
    fd.cloc.assign(T, make_ushort4(0, 0, 0, 0));
    parallel_for(nch, 4, [&](long first, long last) {
        std::vector<int> fq((size_t)kFdChunk * npe2), at;
        for (long ch = first; ch < last; ++ch) {
            const int e0 = (int)ch * kFdChunk, e1 = std::min(T, e0 + kFdChunk);
            Chunk& k = chunk[ch];
            const int* v = &c->h_elem_nodes[(size_t)e0 * npe];
            k.nodes.assign(v, v + (size_t)(e1 - e0) * npe);
            std::sort(k.nodes.begin(), k.nodes.end());
            k.nodes.erase(std::unique(k.nodes.begin(), k.nodes.end()), k.nodes.end());
            // the chunk's part of each node's row, in a dense table: local
            // number of the non-zero, -1 while not met
            at.assign(1, 0);
            for (int i : k.nodes) at.push_back(at.back() + rp[i + 1] - rp[i]);
            std::vector<int> number(at.back(), -1);
            for (int e = e0; e < e1; ++e, v += npe) {
                int l[4] = {0, 0, 0, 0};
                for (int j = 0; j < npe; ++j)
                    l[j] = (int)(std::lower_bound(k.nodes.begin(), k.nodes.end(), v[j]) - k.nodes.begin());
                fd.cloc[e] = make_ushort4((unsigned short)l[0], (unsigned short)l[1], (unsigned short)l[2],
                                          (unsigned short)l[3]);
                for (int m = 0; m < npe; ++m)
                    for (int r = 0; r < npe; ++r) {
                        const int i = v[r], q = (int)(std::lower_bound(&cl[rp[i]], &cl[0] + rp[i + 1], v[m]) - &cl[0]);
                        int& n = number[at[l[r]] + q - rp[i]];
                        if (n < 0) {
                            n = (int)k.qs.size();
                            k.qs.push_back(q);
                            k.cnt.push_back(0);
                        }
                        k.cnt[n]++;
                        fq[(size_t)(e - e0) * npe2 + m * npe + r] = n;
                    }
            }
            k.pos.assign(k.qs.size() + 1, 0);
            for (size_t p = 0; p < k.qs.size(); ++p) k.pos[p + 1] = k.pos[p] + k.cnt[p];
            std::vector<int> next(k.pos.begin(), k.pos.end() - 1);
            k.slots.resize((size_t)(e1 - e0) * npe2);
            for (int e = 0; e < e1 - e0; ++e)
                for (int t = 0; t < npe2; ++t)
                    k.slots[next[fq[(size_t)e * npe2 + t]]++] = (unsigned short)(t * kFdChunk + e);
        }
    });
    // chunks touching each non-zero, and the places of the shared ones'
    // partials (non-zero-major, ascending chunk)
    std::vector<int> nchunk(P->nnz, 0), place(P->nnz, -1);
    for (const Chunk& k : chunk)
        for (int q : k.qs) nchunk[q]++;
    fd.sptr.assign(1, 0);
    for (int q = 0; q < P->nnz; ++q)
        if (nchunk[q] > 1) {
            place[q] = fd.sptr.back();
            fd.shared.push_back(make_int4(q, lu_dst[q], 0, 2 * rowof[q] + (cl[q] == rowof[q] ? 1 : 0)));
            fd.sptr.push_back(fd.sptr.back() + nchunk[q]);
        }
    parallel_for(nch, 4, [&](long first, long last) {
        std::vector<int> asc, rank, order, hist;
        for (long ch = first; ch < last; ++ch) {
            Chunk& k = chunk[ch];
            // the sums' places: finished non-zeros, then shared ones, ascending
            const int np = (int)k.qs.size();
            asc.resize(np);
            for (int p = 0; p < np; ++p) asc[p] = p;
            std::sort(asc.begin(), asc.end(), [&](int x, int y) {
                const bool sx = nchunk[k.qs[x]] > 1, sy = nchunk[k.qs[y]] > 1;
                return sx != sy ? sy : k.qs[x] < k.qs[y];
            });
            rank.resize(np);
            for (int r = 0; r < np; ++r) {
                const int q = k.qs[asc[r]], i = rowof[q];
                rank[asc[r]] = r;
                if (nchunk[q] > 1) {
                    k.shared.push_back(q);
                } else {
                    const int li = (int)(std::lower_bound(k.nodes.begin(), k.nodes.end(), i) - k.nodes.begin());
                    k.done.push_back(make_int4(q, lu_dst[q], 0, 2 * li + (cl[q] == i ? 1 : 0)));
                }
            }
            // the non-zeros by falling number of slots (a counting sort)
            const int most = *std::max_element(k.cnt.begin(), k.cnt.end());
            hist.assign(most + 2, 0);
            for (int p = 0; p < np; ++p) hist[most - k.cnt[p] + 1]++;
            for (int n = 0; n <= most; ++n) hist[n + 1] += hist[n];
            order.resize(np);
            for (int p = 0; p < np; ++p) order[hist[most - k.cnt[p]]++] = p;
            std::vector<unsigned short>& list = k.list;
            const int ng = k.ng = (np + 31) / 32;
            list.resize(fd_list_offs(ng), 0);
            for (int g = 0; g < ng; ++g) list[g + 1] = (unsigned short)(list[g] + k.cnt[order[32 * g]]);
            // lanes past the last non-zero leave their zero past the sums
            for (int r = 0; r < 32 * ng; ++r) list.push_back((unsigned short)(r < np ? rank[order[r]] : r));
            for (int g = 0; g < ng; ++g) {
                const size_t base = list.size();
                list.resize(base + 32 * (size_t)k.cnt[order[32 * g]], (unsigned short)(npe2 * kFdChunk));
                for (int l = 0; l < 32 && 32 * g + l < np; ++l) {
                    const int p = order[32 * g + l];
                    for (int t = 0; t < k.cnt[p]; ++t) list[base + 32 * (size_t)t + l] = k.slots[k.pos[p] + t];
                }
            }
        }
    });
    fd.cnode_ptr.assign(1, 0);
    fd.done_ptr.assign(1, 0);
    fd.share_ptr.assign(1, 0);
    size_t words = 0, nodes = 0, done = 0;
    for (const Chunk& k : chunk) {
        words += k.list.size();
        nodes += k.nodes.size();
        done += k.done.size();
    }
    if (words / 8 >= (size_t)INT32_MAX) throw Error("difference quotients: mesh too large");
    fd.list.reserve(words);
    fd.cnode.reserve(nodes);
    fd.done.reserve(done);
    fd.share.reserve(fd.sptr.back());
    for (const Chunk& k : chunk) {
        fd.nnmax = std::max(fd.nnmax, (int)k.nodes.size());
        fd.cnode.insert(fd.cnode.end(), k.nodes.begin(), k.nodes.end());
        fd.cnode_ptr.push_back((int)fd.cnode.size());
        fd.done.insert(fd.done.end(), k.done.begin(), k.done.end());
        fd.done_ptr.push_back((int)fd.done.size());
        for (int q : k.shared) fd.share.push_back(place[q]++);
        fd.share_ptr.push_back((int)fd.share.size());
        fd.list_at.push_back(make_int2((int)(fd.list.size() / 8), k.ng));
        fd.list.insert(fd.list.end(), k.list.begin(), k.list.end());
        fd.list_max = std::max(fd.list_max, (int)k.list.size());
        fd.grp_max = std::max(fd.grp_max, k.ng);
    }
    fd.list_at.push_back(make_int2((int)(fd.list.size() / 8), 0));
}

static void build_pattern(fvm_ctx* c, BlockILU* P) {
    const int N = c->N, npe = c->npe, T = c->T;
    // node -> elements (host copy of the incidence lists)
    std::vector<int> inc_ptr(N + 1, 0), inc((size_t)T * npe);
    for (size_t q = 0; q < (size_t)T * npe; ++q) inc_ptr[c->h_elem_nodes[q] + 1]++;
    for (int i = 0; i < N; ++i) inc_ptr[i + 1] += inc_ptr[i];
    {
        std::vector<int> pos(inc_ptr.begin(), inc_ptr.end() - 1);
        for (int e = 0; e < T; ++e)
            for (int k = 0; k < npe; ++k) inc[pos[c->h_elem_nodes[(size_t)e * npe + k]]++] = e;
    }
    // pattern: node i couples to every node of every element containing i
    P->h_rowptr.assign(N + 1, 0);
    auto row_of = [&](int i, std::vector<int>& row) {
        row.clear();
        for (int p = inc_ptr[i]; p < inc_ptr[i + 1]; ++p)
            for (int k = 0; k < npe; ++k) row.push_back(c->h_elem_nodes[(size_t)inc[p] * npe + k]);
        std::sort(row.begin(), row.end());
        row.erase(std::unique(row.begin(), row.end()), row.end());
    };
    // (counted and formed in two passes: the rows' places follow from the counts)
    parallel_for(N, 512, [&](long first, long last) {
        std::vector<int> row;
        for (long i = first; i < last; ++i) {
            row_of((int)i, row);
            P->h_rowptr[i + 1] = (int)row.size();
        }
    });
    for (int i = 0; i < N; ++i) P->h_rowptr[i + 1] += P->h_rowptr[i];
    P->nnz = P->h_rowptr[N];
    P->h_col.resize(P->nnz);
    parallel_for(N, 512, [&](long first, long last) {
        std::vector<int> row;
        for (long i = first; i < last; ++i) {
            row_of((int)i, row);
            std::copy(row.begin(), row.end(), P->h_col.begin() + P->h_rowptr[i]);
        }
    });
    const std::vector<int>& rp = P->h_rowptr;
    const std::vector<int>& cl = P->h_col;
    std::vector<int> rowof(P->nnz);
    for (int i = 0; i < N; ++i)
        for (int p = rp[i]; p < rp[i + 1]; ++p) rowof[p] = i;
    // blocks of contiguous nodes; on a large mesh a multiple of the SM count
    // (c->ilu_per_sm blocks per SM: fewer, larger blocks precondition better,
    // more, smaller ones have shorter level chains and share an SM)
    int nsm = 148;
    FVM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device));
    int target = 1500;
    int nb;
    // per_sm 0 (the default): the fewest blocks per SM that keep a block at
    // most kAutoBlockRows rows, the size whose FP32 factor window still fits
    // the staged apply's shared memory (1 on the 200k-node box, 5 at 1M)
    constexpr double kAutoBlockRows = 1600.0;
    const int per_sm = c->ilu_per_sm > 0 ? c->ilu_per_sm
                                         : std::max(1, (int)std::ceil((double)N / (nsm * kAutoBlockRows)));
    if (N >= nsm * 256) nb = nsm * per_sm;
    else nb = std::max(1, (N + target - 1) / target);
    nb = std::min(nb, N);
    std::vector<int> bstart(nb + 1);
    for (int b = 0; b <= nb; ++b) bstart[b] = (int)(((long)N * b) / nb);
    int maxb = 0;
    for (int b = 0; b < nb; ++b) maxb = std::max(maxb, bstart[b + 1] - bstart[b]);
    if (maxb > 65535) throw Error("block-ILU: block too large");
    // Inside each block the factor works in a colour order: a greedy
    // colouring of the block's rows (natural order, smallest colour unused
    // by an earlier neighbour in the block), rows sorted by (colour, row).
    // No two rows of one colour are coupled, so each triangular sweep has as
    // many levels as colours (8 on the tetrahedral meshes, against about 33
    // in natural order).  Position r0 + ii of the factor is global row
    // lu_row[r0 + ii].
    std::vector<int> lu_ptr(N + 1, 0), lu_src, lu_diag(N), lu_row(N);
    std::vector<unsigned short> lu_col;
    std::vector<int> lvl(N), ulvl(N);
    // rows by level, a block's in [r0, r1); a block's levels end at its runs of
    // lvl_ptr (from blk_lvl on)
    std::vector<int> lvl_ptr(1, 0), lvl_rows(N), blk_lvl(1, 0), ulvl_ptr(1, 0), ulvl_rows(N), blk_ulvl(1, 0);
    int nlmax = 0;
    // Schur coupling: interface rows last, levels split by group, and the
    // off-block entries of each factor position
    P->schur_iters = c->schur_iters;
    const bool schur = P->schur_iters >= 0;
    std::vector<int> sch_lv(2 * (size_t)nb, 0), sch_nin(nb, 0), o_ptr(N + 1, 0), o_col, o_src;
    std::vector<std::vector<int>> ends(nb), uends(nb);
    const long grain = std::max(1l, 1024l * nb / N);   // blocks that are worth a thread (0.1 ms each of its uses)
    parallel_for(nb, grain, [&](long first, long last) {
        for (long b = first; b < last; ++b) {
            const int r0 = bstart[b], r1 = bstart[b + 1];
            int nin = r1 - r0;
            const std::vector<int> ord = block_colour_order(rp, cl, r0, r1, schur, &nin);
            sch_nin[b] = nin;
            for (int ii = 0; ii < r1 - r0; ++ii) {
                const int i = r0 + ord[ii];
                lu_row[r0 + ii] = i;
                int inside = 0;
                for (int p = rp[i]; p < rp[i + 1]; ++p) inside += cl[p] >= r0 && cl[p] < r1;
                lu_ptr[r0 + ii + 1] = inside;
                if (schur) o_ptr[r0 + ii + 1] = rp[i + 1] - rp[i] - inside;
            }
        }
    });
    for (int q = 0; q < N; ++q) {
        lu_ptr[q + 1] += lu_ptr[q];
        o_ptr[q + 1] += o_ptr[q];
    }
    lu_src.resize(lu_ptr[N]);
    lu_col.resize(lu_ptr[N]);
    o_col.resize(o_ptr[N]);
    o_src.resize(o_ptr[N]);
    parallel_for(nb, grain, [&](long first, long last) {
        for (long b = first; b < last; ++b) {
            const int r0 = bstart[b], r1 = bstart[b + 1], nin = sch_nin[b];
            std::vector<int> linv(r1 - r0);
            for (int q = r0; q < r1; ++q) linv[lu_row[q] - r0] = q - r0;
            std::vector<std::pair<int, int>> ent;
            for (int q = r0; q < r1; ++q) {
                const int i = lu_row[q];
                ent.clear();
                int o = o_ptr[q];
                for (int p = rp[i]; p < rp[i + 1]; ++p) {
                    const int j = cl[p];
                    if (j >= r0 && j < r1) {
                        ent.emplace_back(linv[j - r0], p);
                    } else if (schur) {
                        o_col[o] = j;
                        o_src[o++] = p;
                    }
                }
                std::sort(ent.begin(), ent.end());
                lu_diag[q] = -1;
                int at = lu_ptr[q];
                for (auto& e : ent) {
                    if (e.first == q - r0) lu_diag[q] = at;
                    lu_src[at] = e.second;
                    lu_col[at++] = (unsigned short)e.first;
                }
                if (lu_diag[q] < 0) throw Error("block-ILU: missing diagonal");
            }
            // with the Schur coupling no level mixes interior and interface
            // rows: forward, every interface row comes after the last interior
            // level; backward, every interior row after the last interface level
            int nl = 0, lvB = 0;
            for (int i = r0; i < r1; ++i) {
                int l = 0;
                for (int p = lu_ptr[i]; p < lu_diag[i]; ++p) l = std::max(l, lvl[r0 + lu_col[p]] + 1);
                if (schur && i - r0 >= nin) l = std::max(l, lvB);
                lvl[i] = l;
                nl = std::max(nl, l + 1);
                if (i - r0 < nin) lvB = nl;
            }
            int nu = 0, uvS = 0;
            for (int i = r1 - 1; i >= r0; --i) {
                int l = 0;
                for (int p = lu_diag[i] + 1; p < lu_ptr[i + 1]; ++p) l = std::max(l, ulvl[r0 + lu_col[p]] + 1);
                if (schur && i - r0 < nin) l = std::max(l, uvS);
                ulvl[i] = l;
                nu = std::max(nu, l + 1);
                if (i - r0 >= nin) uvS = nu;
            }
            sch_lv[2 * (size_t)b] = lvB;
            sch_lv[2 * (size_t)b + 1] = uvS;
            // rows by level, ascending in each
            auto by_level = [&](const std::vector<int>& level, int n, std::vector<int>& rows, std::vector<int>& end) {
                end.assign(n + 1, 0);
                for (int i = r0; i < r1; ++i) end[level[i] + 1]++;
                for (int l = 0; l < n; ++l) end[l + 1] += end[l];
                std::vector<int> next(end.begin(), end.end() - 1);
                for (int i = r0; i < r1; ++i) rows[r0 + next[level[i]]++] = i;
            };
            by_level(lvl, nl, lvl_rows, ends[b]);
            by_level(ulvl, nu, ulvl_rows, uends[b]);
        }
    });
    for (int b = 0; b < nb; ++b) {
        nlmax = std::max(nlmax, (int)std::max(ends[b].size(), uends[b].size()) - 1);
        for (size_t l = 1; l < ends[b].size(); ++l) lvl_ptr.push_back(bstart[b] + ends[b][l]);
        for (size_t l = 1; l < uends[b].size(); ++l) ulvl_ptr.push_back(bstart[b] + uends[b][l]);
        blk_lvl.push_back((int)lvl_ptr.size() - 1);
        blk_ulvl.push_back((int)ulvl_ptr.size() - 1);
    }
    P->nb = nb;
    P->maxb = maxb;
    P->nlevels_max = nlmax;
    // the layout of every block's factor and its record
    std::vector<IluBlk> blk(nb);
    std::vector<std::vector<unsigned short>> bmeta(nb), bcol(nb);
    IluPlaces at;
    at.entry.resize(lu_src.size());
    at.upper.resize(N);
    at.lower.resize(N);
    parallel_for(nb, grain, [&](long b0, long b1) {
        for (long b = b0; b < b1; ++b) {
            blk[b] = ilu_layout(bstart[b], bstart[b + 1], lu_ptr, lu_diag, lu_col,
                                {lvl_ptr, lvl_rows, blk_lvl[b], blk_lvl[b + 1]},
                                {ulvl_ptr, ulvl_rows, blk_ulvl[b], blk_ulvl[b + 1]}, at, bmeta[b], bcol[b]);
            blk[b].seg = blk_lvl[b];
        }
    });
    const std::vector<int>& spos = at.entry;
    std::vector<unsigned short> meta, scol;
    size_t nlu = 0;
    for (int b = 0; b < nb; ++b) {
        blk[b].v0 = (int)nlu;
        blk[b].c0 = (int)scol.size();
        blk[b].mo = (int)meta.size();
        nlu += ilu_window(bstart[b + 1] - bstart[b], blk[b].ds);
        scol.insert(scol.end(), bcol[b].begin(), bcol[b].end());
        meta.insert(meta.end(), bmeta[b].begin(), bmeta[b].end());
        if (nlu >= (size_t)INT32_MAX || scol.size() >= (size_t)INT32_MAX || meta.size() >= (size_t)INT32_MAX)
            throw Error("block-ILU: block too large");
    }
    P->nlu = nlu;
    for (int b = 0; b < nb; ++b) P->wide = P->wide || blk[b].nwide > 0;
    // elimination schedule in level order (window positions relative to each
    // block's first entry, as the factorisation indexes); the same update set
    // and order as merging row i with U(k) for each L entry
    std::vector<int> seg_ptr(lvl_ptr.size(), 0);
    std::vector<std::vector<unsigned>> bupd(nb);
    parallel_for(nb, grain, [&](long b0, long b1) {
        for (long b = b0; b < b1; ++b) {
            const int r0 = bstart[b];
            std::vector<unsigned>& u = bupd[b];
            for (int g = blk_lvl[b]; g < blk_lvl[b + 1]; ++g) {
                const int q0 = lvl_ptr[g], q1 = lvl_ptr[g + 1];
                const size_t head = u.size();
                u.resize(head + at.lower[lvl_rows[q1 - 1]] / kIluGroup * kIluGroup + kIluGroup, 0u);
                for (int q = q0; q < q1; ++q) {
                    const int i = lvl_rows[q];
                    u[head + at.lower[i]] = (unsigned)(u.size() - head);
                    for (int p = lu_ptr[i]; p < lu_diag[i]; ++p) {
                        const size_t cw = u.size();
                        u.push_back(0u);
                        const int k = r0 + lu_col[p];
                        int kpos = lu_diag[k] + 1;
                        const int kend = lu_ptr[k + 1];
                        for (int jj = p + 1; jj < lu_ptr[i + 1] && kpos < kend; ++jj) {
                            const int j = lu_col[jj];
                            while (kpos < kend && lu_col[kpos] < j) ++kpos;
                            if (kpos < kend && lu_col[kpos] == j)
                                u.push_back((unsigned)spos[jj] | ((unsigned)spos[kpos] << 16));
                        }
                        u[cw] = (unsigned)(u.size() - cw - 1);
                    }
                }
                seg_ptr[g + 1] = (int)(u.size() - head);
            }
        }
    });
    std::vector<unsigned> upd;
    size_t seg_max = 0, nupd = 0;
    for (const auto& u : bupd) nupd += u.size();
    if (nupd >= (size_t)INT32_MAX) throw Error("block-ILU: elimination schedule too large");
    upd.reserve(nupd);
    for (const auto& u : bupd) upd.insert(upd.end(), u.begin(), u.end());
    for (size_t g = 0; g + 1 < seg_ptr.size(); ++g) {
        seg_max = std::max(seg_max, (size_t)seg_ptr[g + 1]);
        seg_ptr[g + 1] += seg_ptr[g];
    }
    {
        size_t need64 = 0, need32 = 0, exact64 = 0, exact32 = 0;
        bool fits16 = true, exact16 = true;
        for (int b = 0; b < nb; ++b) {
            const size_t nr = bstart[b + 1] - bstart[b], ds = blk[b].ds;
            // the schedule's window positions and the columns are 16-bit words
            if (ilu_window(nr, ds) >= 65536 || nr + 1 >= 65535) fits16 = false;
            for (size_t sz : {(size_t)8, (size_t)4}) {
                const size_t need = ilu_stage_bytes(nr, ds, blk[b].mw, sz);
                if (sz == 8) need64 = std::max(need64, need);
                else need32 = std::max(need32, need);
                // rows end to end: vector, values, 16-bit columns; row pointers, pivots'
                // places, rows of the two sweeps and their levels' ends; mbarrier
                const size_t nnz = (size_t)(lu_ptr[bstart[b + 1]] - lu_ptr[bstart[b]]);
                const size_t words = 4 * nr + (size_t)blk[b].nl + blk[b].nu + 3;
                const size_t e = round16(round16(nr * sz) + nnz * (sz + 2) + round16(2 * words)) + 16;
                if (nnz >= 65535 || nr + 1 >= 65535) exact16 = false;
                if (sz == 8) exact64 = std::max(exact64, e);
                else exact32 = std::max(exact32, e);
            }
        }
        P->smem_stage[0] = (fits16 && need64 <= kMaxDynSmem) ? need64 : 0;
        P->smem_stage[1] = (fits16 && need32 <= kMaxDynSmem) ? need32 : 0;
        // two schedule buffers of scr_words words (at most what the
        // factorisation's threads hold in kIluFactorPre registers each)
        for (int pr = 0; pr < 2; ++pr) {
            const size_t st = round16(P->smem_stage[pr]);
            const size_t room = P->smem_stage[pr] && st < kMaxDynSmem ? (kMaxDynSmem - st) / 8 : 0;
            P->scr_words[pr] = (int)std::min<size_t>(std::min<size_t>(seg_max, room), (size_t)kIluFactorThreads * kIluFactorPre);
        }
        // one thread per row of the widest level, in whole warps of 128 or 256
        int widest = 0;
        for (size_t g = 0; g + 1 < lvl_ptr.size(); ++g) widest = std::max(widest, lvl_ptr[g + 1] - lvl_ptr[g]);
        for (size_t g = 0; g + 1 < ulvl_ptr.size(); ++g) widest = std::max(widest, ulvl_ptr[g + 1] - ulvl_ptr[g]);
        P->apply_threads = widest > 128 ? 256 : 128;
        // the global-memory apply keeps the block's vector in shared memory
        if (!P->smem_stage[0]) {
            if (ilu_plain_bytes(maxb, sizeof(double)) > kMaxDynSmem)
                throw Error("block-ILU: blocks too large for the FP64 apply (set more blocks per SM)");
            raise_smem_limit(k_ilu_apply<double>, ilu_plain_bytes(maxb, sizeof(double)));
        }
        if (!P->smem_stage[1]) {
            if (ilu_plain_bytes(maxb, sizeof(float)) > kMaxDynSmem)
                throw Error("block-ILU: blocks too large for the FP32 apply (set more blocks per SM)");
            raise_smem_limit(k_ilu_apply<float>, ilu_plain_bytes(maxb, sizeof(float)));
        }
        if (P->smem_stage[0]) {
            raise_smem_limit(P->wide ? k_ilu_apply_smem<double, true> : k_ilu_apply_smem<double, false>, P->smem_stage[0]);
            raise_smem_limit(k_ilu_factor_smem<double>, (size_t)(round16(P->smem_stage[0]) + 8 * (size_t)P->scr_words[0]));
        }
        if (P->smem_stage[1]) {
            raise_smem_limit(P->wide ? k_ilu_apply_smem<float, true> : k_ilu_apply_smem<float, false>, P->smem_stage[1]);
            raise_smem_limit(k_ilu_factor_smem<float>, (size_t)(round16(P->smem_stage[1]) + 8 * (size_t)P->scr_words[1]));
        }
        if (schur) {
            schur_layout(c, P, 0, exact16 && exact64 <= kMaxDynSmem ? exact64 : 0);
            schur_layout(c, P, 1, exact16 && exact32 <= kMaxDynSmem ? exact32 : 0);
        }
    }
    cudaStream_t s = c->stream;
    if (schur) {
        P->sch_lv.upload(sch_lv, s);
        P->sch_nin.upload(sch_nin, s);
        P->h_sch_nin = sch_nin;
        P->o_ptr.upload(o_ptr, s);
        if (o_col.empty()) { o_col.push_back(0); o_src.push_back(0); }
        P->o_col.upload(o_col, s);
        P->o_src.upload(o_src, s);
        P->xg.alloc(2 * (size_t)N);
        P->sbar.alloc(2);
        P->sbar.zero(s);
        P->serr.alloc(1);
        P->serr.zero(s);
        FVM_CUDA(cudaMallocHost(&P->h_serr, sizeof(int)));
        *P->h_serr = 0;
    }
    P->col.upload(P->h_col, s);
    P->J.alloc(P->nnz);
    {
        std::vector<int> lu_pos(N);
        for (int q = 0; q < N; ++q) lu_pos[lu_row[q]] = q;
        P->lu_pos.upload(lu_pos, s);
    }
    P->fd_g.alloc((size_t)c->nz * N);
    P->fd_dg.alloc((size_t)c->nz * N);
    P->fd_gq.alloc((size_t)c->nz * N);
    P->fd_diag.alloc(N);
    {
        // 1/V of free rows, 0 on Dirichlet rows
        std::vector<double> sc(N);
        FVM_CUDA(cudaMemcpyAsync(sc.data(), c->invV.p, sizeof(double) * N, cudaMemcpyDeviceToHost, s));
        FVM_CUDA(cudaStreamSynchronize(s));
        for (int i = 0; i < N; ++i)
            if (c->h_node_type[i]) sc[i] = 0.0;
        P->fd_scale.upload(sc, s);
        FVM_CUDA(cudaStreamSynchronize(s));
    }
    P->ahhp.alloc(N);
    P->rowptr.upload(P->h_rowptr, s);
    P->bstart.upload(bstart, s);
    P->h_bstart = bstart;
    P->h_lu_row = lu_row;
    {
        // where the quotient kernels put each Jacobian entry for the factorisation
        std::vector<int> lu_dst(P->nnz, -1);
        for (int b = 0; b < nb; ++b)
            for (int p = lu_ptr[bstart[b]]; p < lu_ptr[bstart[b + 1]]; ++p) lu_dst[lu_src[p]] = blk[b].v0 + spos[p];
        FdTables fd;
        build_fd_tables(c, P, rowof, lu_dst, fd);
        P->fd_cnode_ptr.upload(fd.cnode_ptr, s);
        P->fd_cnode.upload(fd.cnode, s);
        P->fd_cloc.upload(fd.cloc, s);
        P->fd_list_at.upload(fd.list_at, s);
        P->fd_list.upload(fd.list, s);
        P->fd_done_ptr.upload(fd.done_ptr, s);
        P->fd_done.upload(fd.done, s);
        P->fd_share_ptr.upload(fd.share_ptr, s);
        P->fd_share.upload(fd.share, s);
        P->fd_shared.upload(fd.shared, s);
        P->fd_sptr.upload(fd.sptr, s);
        P->fd_part.alloc(fd.sptr.back());
        P->fd_nnmax = fd.nnmax;
        P->fd_list_max = fd.list_max;
        P->fd_grp_max = fd.grp_max;
        // the tables' host memory is read by copies still in flight
        FVM_CUDA(cudaStreamSynchronize(s));
    }
    P->blk.upload(blk, s);
    if (!P->smem_stage[0] || !P->smem_stage[1]) P->lu_up.upload(at.upper, s);
    P->lu_row.upload(lu_row, s);
    P->lu_col.upload(scol, s);
    if (upd.empty()) upd.push_back(0u);
    P->seg_ptr.upload(seg_ptr, s);
    P->upd.upload(upd, s);
    P->meta.upload(meta, s);
    P->status.alloc(1);
    P->status.zero(s);
    FVM_CUDA(cudaMallocHost(&P->h_status, sizeof(int)));
    FVM_CUDA(cudaStreamSynchronize(s));
    P->built = true;
}

// fills in the operator layout's places of the quotient kernels' outputs
__global__ void k_fd_op_places(int n, int4* __restrict__ at, const int* __restrict__ op_dst) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) at[t].z = op_dst[at[t].x];
}
void fd_set_op_places(fvm_ctx* c, const std::vector<int>& op_dst) {
    BlockILU* P = c->ilu;
    DevBuf<int> d;
    d.upload(op_dst, c->stream);
    for (DevBuf<int4>* b : {&P->fd_done, &P->fd_shared})
        if (b->n) fvm_launch(c, k_fd_op_places, grid_for((long)b->n, 256), 256, 0, c->stream, (int)b->n, b->p, d.p);
    FVM_CUDA(cudaStreamSynchronize(c->stream));
}

void psetup_dev(fvm_ctx* c, double cj, double h, const double* y, const double* yp,
                const double* F0, const double* ewt, int precision) {
    if (!c->ilu) c->ilu = new BlockILU();
    BlockILU* P = c->ilu;
    if (!P->built) build_pattern(c, P);
    cudaStream_t s = c->stream;
    const int N = c->N;
    c->tm.begin(TM_FD_JAC, s);
    FVM_CUDA(cudaMemsetAsync(P->status.p, 0, sizeof(int), s));
    (void)F0;   // the element-wise quotients difference each element's own partials
    // the fused cycle's operator values too, once its layout exists
    const bool op = P->op_built && P->fused_ok;
    fvm_launch_pdl(c, k_fd_node, grid_for(N, 256), 256, 0, s, N, y, yp, ewt, h, std::sqrt(DBL_EPSILON), cj, c->zones.p,
               c->nz, c->nz_ptr.p, c->nz_zone.p, c->nz_w.p, c->rho0, c->ntype.p, c->hD.p,
               FdNode{P->fd_g.p, P->fd_dg.p, P->fd_gq.p, P->fd_diag.p, P->ahhp.p, op ? P->op_dg.p : nullptr,
                      P->lu_pos.p});
    P->cj_setup = cj;
    P->setup_id++;
    P->op_setup_id = op ? P->setup_id : -1;
    {
        FdArgs a;
        a.T = c->T; a.N = N; a.kiso = c->kiso ? 1 : 0; a.estride = c->estride; a.nnmax = P->fd_nnmax;
        a.cnode_ptr = P->fd_cnode_ptr.p; a.cnode = P->fd_cnode.p; a.cloc = P->fd_cloc.p;
        a.list_at = P->fd_list_at.p; a.list = reinterpret_cast<const uint4*>(P->fd_list.p);
        a.done_ptr = P->fd_done_ptr.p; a.done = P->fd_done.p; a.share_ptr = P->fd_share_ptr.p; a.share = P->fd_share.p;
        a.list_max = P->fd_list_max; a.grp_max = P->fd_grp_max; a.part = P->fd_part.p;
        a.coef = c->coef.p; a.xyz = c->xyz.p; a.eK = c->eK.p; a.ezone = c->ezone.p;
        a.y = y; a.g = P->fd_g.p; a.dg = P->fd_dg.p; a.gq = P->fd_gq.p; a.upw = c->upw.p;
        // one buffer per precision: the groups' padding stays zero in each
        auto window = [&](auto& w) -> void* {
            if (!w.n) {
                w.alloc(P->nlu);
                w.zero(s);
            }
            return w.p;
        };
        a.out = FdOut{P->fd_scale.p, P->fd_diag.p, P->J.p, precision ? window(P->Jw32) : window(P->Jw),
                      op ? P->op_val.p : nullptr};
        auto run = [&](auto one) {
            using S = decltype(one);
            auto go = [&](auto kern, size_t sm) {
                if (sm > 48 * 1024) raise_smem_limit(kern, sm);
                fvm_launch_pdl(c, kern, (c->T + kFdChunk - 1) / kFdChunk, kFdThreads, sm, s, a);
            };
#define FVM_FD(NPE, NFE, RC, MZ) \
    go(k_fd_chunk<NPE, NFE, RC, MZ, S>, FdSmem(NPE, RC, MZ, sizeof(S), a.nnmax, a.list_max, a.grp_max).bytes)
            const bool mz = c->nz > 1;
            if (c->dim == 2) mz ? FVM_FD(3, 3, false, true) : FVM_FD(3, 3, false, false);
            else if (c->recompute) mz ? FVM_FD(4, 6, true, true) : FVM_FD(4, 6, true, false);
            else mz ? FVM_FD(4, 6, false, true) : FVM_FD(4, 6, false, false);
#undef FVM_FD
            const int ns = (int)P->fd_shared.n;
            if (ns)
                fvm_launch_pdl(c, k_fd_shared<S>, grid_for(ns, 256), 256, 0, s, ns, P->fd_shared.p, P->fd_sptr.p,
                           P->fd_part.p, a.out);
        };
        if (precision) run(0.f);
        else run(0.0);
    }
    c->tm.end(TM_FD_JAC, s);
    c->tm.begin(TM_ILU_FACTOR, s);
    auto factor = [&](auto& lu, auto* Jw) {
        using T = std::remove_pointer_t<decltype(Jw)>;
        lu.alloc(P->nlu + kIluSlack);   // a sweep in place may read past the last block's
        if (P->smem_stage[precision]) {
            const int so = (int)round16(P->smem_stage[precision]);
            const int sw = P->scr_words[precision];
            fvm_launch_pdl(c, k_ilu_factor_smem<T>, P->nb, kIluFactorThreads, (size_t)so + 8 * (size_t)sw, s, P->bstart.p,
                       P->blk.p, P->meta.p, (const T*)Jw, P->lu_col.p, P->seg_ptr.p, P->upd.p, so, sw, lu.p,
                       P->status.p);
        } else {
            fvm_launch(c, k_ilu_factor<T>, P->nb, kIluPlainFactorThreads, 0, s, P->bstart.p, P->blk.p, P->meta.p, P->lu_up.p,
                       (const T*)Jw, P->lu_col.p, lu.p, P->status.p);
        }
    };
    if (precision) factor(P->lu32, P->Jw32.p);
    else factor(P->lu64, P->Jw.p);
    c->tm.end(TM_ILU_FACTOR, s);
    // (also what keeps an apply's early reads of the factor behind the kernel above,
    // which lets its successor start before it factors: fvm_launch_pdl)
    FVM_CUDA(cudaMemcpyAsync(P->h_status, P->status.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    P->factored = precision;
}

void jacobian_apply(fvm_ctx* c, double cj, const double* x, double* y, const int* skip, const double* dcj_dev) {
    BlockILU* P = c->ilu;
    if (!P || P->factored < 0) throw Error("jacobian_apply: preconditioner not set up");
    fvm_launch_pdl(c, k_jac_apply, grid_for(4L * c->N, 256), 256, 0, c->stream, c->N, P->rowptr.p, P->col.p,
                   P->J.p, P->ahhp.p, c->ntype.p, cj - P->cj_setup, x, y, skip, dcj_dev);
}

double jacobian_cj_setup(fvm_ctx* c) { return c->ilu ? c->ilu->cj_setup : 0.0; }
int ilu_factored(fvm_ctx* c) { return c->ilu ? c->ilu->factored : -1; }
bool schur_active(fvm_ctx* c) { return c->ilu && c->ilu->schur_iters >= 0; }

int ilu_status(fvm_ctx* c) {
    if (!c->ilu || !c->ilu->h_status) return 0;
    ctx_sync(c);
    return *c->ilu->h_status;
}

int ilu_status_seen(fvm_ctx* c) { return c->ilu && c->ilu->h_status ? *c->ilu->h_status : 0; }

const int* ilu_status_dev(fvm_ctx* c) { return c->ilu ? c->ilu->status.p : nullptr; }

bool ilu_ready(fvm_ctx* c) { return c->ilu && c->ilu->factored >= 0; }

int schur_status(fvm_ctx* c) {
    BlockILU* P = c->ilu;
    if (!P || P->schur_iters < 0 || !P->h_serr) return 0;
    FVM_CUDA(cudaMemcpyAsync(P->h_serr, P->serr.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    ctx_sync(c);
    const int e = *P->h_serr;
    if (e) FVM_CUDA(cudaMemsetAsync(P->serr.p, 0, sizeof(int), c->stream));
    return e;
}

void psolve_dev(fvm_ctx* c, const double* r, double* z, const int* skip) {
    BlockILU* P = c->ilu;
    if (!P || P->factored < 0) throw Error("psolve: preconditioner not set up");
    cudaStream_t s = c->stream;
    c->tm.begin(TM_ILU_APPLY, s);
    struct EndTimer {
        fvm_ctx* c;
        ~EndTimer() { c->tm.end(TM_ILU_APPLY, c->stream); }
    } end_timer{c};
    if (P->schur_iters >= 0) {
        if (!P->schur_smem[P->factored])
            throw Error("psolve: the Schur coupling needs every block's factor and forward result in shared "
                        "memory with all blocks resident at once (use the FP32 factor on large blocks)");
        if (P->factored) launch_schur_apply(c, P, P->lu32.p, r, z, skip);
        else launch_schur_apply(c, P, P->lu64.p, r, z, skip);
        return;
    }
    const size_t sm = P->smem_stage[P->factored];
    auto go = [&](auto staged, auto plain, const auto* lu) {
        if (sm)
            fvm_launch_pdl(c, staged, P->nb, P->apply_threads, sm, s, P->bstart.p, P->blk.p, P->lu_col.p, P->meta.p, lu,
                           P->lu_row.p, r, z, P->status.p, skip);
        else
            fvm_launch_pdl(c, plain, P->nb, P->apply_threads, ilu_plain_bytes(P->maxb, sizeof(*lu)), s, P->bstart.p, P->blk.p,
                           P->lu_col.p, P->meta.p, lu, P->lu_row.p, r, z, skip);
    };
    if (P->factored) go(P->wide ? k_ilu_apply_smem<float, true> : k_ilu_apply_smem<float, false>, k_ilu_apply<float>, P->lu32.p);
    else go(P->wide ? k_ilu_apply_smem<double, true> : k_ilu_apply_smem<double, false>, k_ilu_apply<double>, P->lu64.p);
}

} // namespace fvmb

using namespace fvmb;

void fvmb_destroy_ilu(fvmb::BlockILU* p) {
    if (!p) return;
    if (p->h_status) cudaFreeHost(p->h_status);
    if (p->h_serr) cudaFreeHost(p->h_serr);
    delete p;
}

extern "C" int fvm_psetup(fvm_ctx* c, double t, double cj, double h, const double* y,
                          const double* yp, const double* F0, const double* ewt, int precision) {
    try {
        (void)t;
        if (!c || !y || !yp || !F0 || !ewt) throw Error("fvm_psetup: null argument");
        if (precision != 0 && precision != 1) throw Error("fvm_psetup: precision must be 0 or 1");
        psetup_dev(c, cj, h, y, yp, F0, ewt, precision);
        FVM_CUDA(cudaGetLastError());
        return ilu_status(c) ? 1 : 0;
    } catch (const Error& ex) {
        set_error(ex.what());
        return ex.code;
    } catch (const std::exception& ex) {
        set_error(ex.what());
        return -1;
    }
}

extern "C" int fvm_psolve(fvm_ctx* c, const double* r, double* z) {
    try {
        if (!c || !r || !z) throw Error("fvm_psolve: null argument");
        psolve_dev(c, r, z);
        FVM_CUDA(cudaGetLastError());
        FVM_CUDA(cudaStreamSynchronize(c->stream));
        if (schur_status(c)) throw Error("fvm_psolve: a grid barrier of the Schur-coupled apply timed out");
        return 0;
    } catch (const Error& ex) {
        set_error(ex.what());
        return ex.code;
    } catch (const std::exception& ex) {
        set_error(ex.what());
        return -1;
    }
}

extern "C" int fvm_set_precond_blocks(fvm_ctx* c, int per_sm) {
    try {
        if (!c) throw Error("fvm_set_precond_blocks: null context");
        if (per_sm < 0 || per_sm > 16)
            throw Error("fvm_set_precond_blocks: blocks per SM must be in [1, 16], or 0 for automatic");
        FVM_CUDA(cudaStreamSynchronize(c->stream));
        c->ilu_per_sm = per_sm;
        if (c->ilu) {
            fvmb_destroy_ilu(c->ilu);
            c->ilu = nullptr;
        }
        return 0;
    } catch (const Error& ex) {
        set_error(ex.what());
        return ex.code;
    } catch (const std::exception& ex) {
        set_error(ex.what());
        return -1;
    }
}

extern "C" int fvm_set_precond_schur(fvm_ctx* c, int iters) {
    try {
        if (!c) throw Error("fvm_set_precond_schur: null context");
        if (iters < -1 || iters > 64) throw Error("fvm_set_precond_schur: iterations must be in [-1, 64]");
        FVM_CUDA(cudaStreamSynchronize(c->stream));
        c->schur_iters = iters;
        if (c->ilu) {
            fvmb_destroy_ilu(c->ilu);
            c->ilu = nullptr;
        }
        return 0;
    } catch (const Error& ex) {
        set_error(ex.what());
        return ex.code;
    } catch (const std::exception& ex) {
        set_error(ex.what());
        return -1;
    }
}

extern "C" int fvm_precond_schur_info(fvm_ctx* c, int* iters, int* interface_rows, int* supported) {
    try {
        if (!c || !c->ilu || !c->ilu->built) throw Error("fvm_precond_schur_info: no preconditioner");
        BlockILU* P = c->ilu;
        if (iters) *iters = P->schur_iters;
        if (interface_rows) {
            long n = 0;
            if (P->schur_iters >= 0)
                for (int b = 0; b < P->nb; ++b) n += P->h_bstart[b + 1] - P->h_bstart[b] - P->h_sch_nin[b];
            *interface_rows = (int)n;
        }
        if (supported) *supported = (P->schur_smem[0] ? 1 : 0) | (P->schur_smem[1] ? 2 : 0);
        return 0;
    } catch (const Error& ex) {
        set_error(ex.what());
        return ex.code;
    } catch (const std::exception& ex) {
        set_error(ex.what());
        return -1;
    }
}

// pattern / partition introspection for tests and the autotuner
extern "C" int fvm_precond_info(fvm_ctx* c, int* nnz, int* ncolours, int* nblocks, int* max_levels) {
    try {
        if (!c || !c->ilu || !c->ilu->built) throw Error("fvm_precond_info: no preconditioner");
        if (nnz) *nnz = c->ilu->nnz;
        if (ncolours) {
            if (!c->ilu->ncol) c->ilu->ncol = count_colours(c->ilu->h_rowptr, c->ilu->h_col);
            *ncolours = c->ilu->ncol;
        }
        if (nblocks) *nblocks = c->ilu->nb;
        if (max_levels) *max_levels = c->ilu->nlevels_max;
        return 0;
    } catch (const std::exception& ex) {
        set_error(ex.what());
        return -1;
    }
}

// copies the assembled Jacobian (CSR, host buffers of the sizes reported
// by fvm_precond_info) for inspection against the oracle
extern "C" int fvm_precond_jacobian(fvm_ctx* c, int* rowptr, int* col, double* val) {
    try {
        if (!c || !c->ilu || !c->ilu->built) throw Error("fvm_precond_jacobian: no preconditioner");
        BlockILU* P = c->ilu;
        if (rowptr) std::copy(P->h_rowptr.begin(), P->h_rowptr.end(), rowptr);
        if (col) std::copy(P->h_col.begin(), P->h_col.end(), col);
        if (val) {
            FVM_CUDA(cudaMemcpyAsync(val, P->J.p, sizeof(double) * P->nnz, cudaMemcpyDeviceToHost, c->stream));
            FVM_CUDA(cudaStreamSynchronize(c->stream));
        }
        return 0;
    } catch (const std::exception& ex) {
        set_error(ex.what());
        return -1;
    }
}
