// Block-ILU(0) preconditioner state and the device helpers of its
// shared-memory ("staged") triangular solves, shared by the preconditioner
// kernels (precond.cu) and the fused Arnoldi kernel (arnoldi_fused.cu).
#pragma once

#include "ctx.cuh"
#include "tc05.cuh"

#include <cstdint>
#include <vector>

namespace fvmb {

// One block's factor: rows in colour order, the off-diagonal entries sliced by
// level for the sweeps.  The rows of a level are taken longest first, 32 to a
// slice (a lane each), and a slice's entries are stored entry-major: entry k
// of lane l at 32 (start + k) + l, padded to the slice's longest row with
// zeros whose column is nr, a slot of the vector that stays zero.  The lower
// sweep's slices come first, then the upper sweep's, then the (inverted)
// pivots in row order.  A warp so reads 32 consecutive values and columns.
// Stored row by row instead, with a row per lane, every read hit about four
// lanes' worth of bank conflicts, and the sweeps were bound by those.
struct IluBlk {
    int v0;    // first entry in the value arrays (a multiple of 32)
    int c0;    // and in the column array
    int dp;    // slices' length / 32: the pivots start at 32 dp
    int mo;    // the record's first word (a multiple of 8)
    int mw;    // its words
    int nl, nu;      // levels of the lower and the upper sweep
    int nsl, nsu;    // their slices
    int seg;     // first level in the elimination schedule
};

struct BlockILU {
    bool built = false;
    int nnz = 0;
    int ncol = 0;             // colours of the reference's set-up, 0 until asked for
    std::vector<int> h_rowptr, h_col;
    DevBuf<int> col;
    DevBuf<double> J;
    // element-wise finite-difference Jacobian: chunks of consecutive elements
    // (the tables of FdTables, precond.cu)
    DevBuf<int> fd_cnode_ptr, fd_cnode, fd_done_ptr, fd_share_ptr, fd_share, fd_sptr;
    DevBuf<int2> fd_list_at;
    DevBuf<int4> fd_done, fd_shared;
    DevBuf<ushort4> fd_cloc;
    DevBuf<unsigned short> fd_list;
    DevBuf<double> fd_part;
    int fd_nnmax = 0, fd_list_max = 0, fd_grp_max = 0;
    DevBuf<int> lu_pos;       // [N] factor position of each node (inverse of lu_row)
    DevBuf<double> fd_g, fd_dg, fd_gq;   // [nz][N] rho0 krw, its change over the shift, their quotient
    DevBuf<double> fd_scale, fd_diag;    // [N] row scale, diagonal subtrahend
    // assembled-operator Krylov products (fvm_opts.krylov_operator = 1):
    // device row pointers of J, the storage coefficient ahh(h + d) behind
    // the cj term of J's diagonal, and the cj of the current set-up
    DevBuf<int> rowptr;
    DevBuf<double> ahhp;
    double cj_setup = 0.0;
    long setup_id = 0;             // set-ups done (the fused operator refreshes after each)
    std::vector<int> h_lu_row, h_bstart;
    // the same operator for the fused Arnoldi kernel: J's rows in factor
    // order, 32 rows per slice (one warp), each slice stored entry-major
    // (entry k of the slice's lane l at slice start + 128 (k / 4) + 4 l + k % 4, rows shorter
    // than the slice's longest padded with zero entries of their own column;
    // four entries of a lane together, OpSlice)
    bool op_built = false, fused_ok = false;
    long op_setup_id = -1;
    DevBuf<int> op_slptr, op_blksl, op_src;
    DevBuf<unsigned short> op_lcol;   // 16-bit columns into each block's node list
    DevBuf<int> halo_ptr, halo_node;           // each block's node list: its rows in factor order, its halo
    DevBuf<int> nbr_ptr, nbr;                  // blocks whose rows a block's operator reads
    DevBuf<unsigned> flags;                    // per block: last step published; the barrier counter
    unsigned fused_launches = 0;               // since the flags were zero
    DevBuf<float> op_val, op_dg;
    size_t fused_smem = 0, fused_smem_d = 0, fused_stage = 0;   // _d without the Hessenberg matrix
    size_t fused_room[2] = {0, 0};           // dynamic shared bytes each variant may have
    bool fused_var_ok[2] = {false, false};   // CGS2 / delayed variant can run
    int fused_threads = 0, fused_nrmax = 0, fused_nhmax = 0, fused_hmax = 0, fused_nqp = 0;
    int nb = 0, maxb = 0;
    DevBuf<int> bstart;
    DevBuf<IluBlk> blk;       // [nb] where each block's factor and records start
    size_t nlu = 0;           // factor entries of all blocks (padding included)
    // the set-up's Jacobian in factor order, for an FP64 and an FP32 factor
    // (written by the quotient kernels; allocated at the first use of each)
    DevBuf<double> Jw;
    DevBuf<float> Jw32;
    DevBuf<int> lu_up;        // [N] lane of each row in the upper slices (blocks not staged)
    DevBuf<int> lu_row;       // global row of each factor position (colour order inside the blocks)
    // ILU(0) elimination schedule of the shared-memory factorisation, one
    // contiguous segment per level (upd[seg_ptr[g] .. seg_ptr[g+1]), g the
    // block's first level (IluBlk::seg) plus the level): the offset of the
    // list of each lane of the level's slices, then per row and per L entry
    // in column order a count word followed by that many (target | source <<
    // 16) window positions
    DevBuf<int> seg_ptr;
    DevBuf<unsigned> upd;
    int scr_words[2] = {0, 0};   // shared-memory schedule scratch of the factorisation (words), by precision
    DevBuf<unsigned short> lu_col;
    DevBuf<unsigned short> meta;   // per-block records of the sweeps (ilu_meta_words)
    DevBuf<double> lu64;
    DevBuf<float> lu32;
    int factored = -1;        // precision of the current factor, -1 none
    DevBuf<int> status;
    int* h_status = nullptr;  // pinned
    int nlevels_max = 0;
    size_t smem_stage[2] = {0, 0};   // staged apply: shared bytes for FP64 / FP32, 0 = not possible
    int apply_threads = 128;         // CTA of the staged apply: 128, or 256 when a level is wider
    // Schur interface coupling (fvm_set_precond_schur; decomp/schur.c):
    // each block's interface rows (coupled to another block) follow its
    // interior rows in the factor; the forward levels [0, lvB) of a block
    // hold only interior rows and the rest only interface rows, the
    // backward levels [0, uvS) only interface rows and the rest only
    // interior rows (sch_lv[2b] = lvB, sch_lv[2b+1] = uvS, sch_nin[b] =
    // interior rows).  o_ptr/o_col/o_src: the off-block entries of each
    // factor position (global column, index into J), ascending column.
    int schur_iters = -1;
    DevBuf<int> sch_lv, sch_nin, o_ptr, o_col, o_src;
    std::vector<int> h_sch_nin;
    DevBuf<double> xg;               // 2 N: published interface iterates (node order), by parity
    DevBuf<unsigned> sbar;           // grid barrier of the coupled apply
    DevBuf<int> serr;                // 3: a grid barrier of the coupled apply timed out
    int* h_serr = nullptr;           // pinned
    size_t schur_smem[2] = {0, 0};   // dynamic shared bytes of the coupled apply, 0 = not possible
    int schur_nrmax = 0;
};

// largest dynamic shared-memory carve-out a CTA may request on sm_100
constexpr size_t kMaxDynSmem = 227 * 1024;
// threads of a staged triangular-solve CTA: levels hold a few dozen rows,
// so a small CTA keeps the per-level barrier cheap
constexpr int kIluThreads = 256;   // largest CTA of the staged apply

// Staged variant: the CTA first brings its block's factor into shared
// memory, then runs the level loops entirely there, so each level costs a
// few shared-memory latencies and a barrier instead of a dependent chain of
// L2/HBM loads.  The block's values, columns and record are each one
// contiguous 16-byte aligned range, moved by 1D TMA bulk copies
// (cp.async.bulk, completion counted on an mbarrier, bounded wait), while the
// threads fill the right-hand side alongside.
// Shared layout: x[T nr + 1, 16-B padded] | val[T wn] | col[u16 32 dp + slack] |
// record | mbarrier (a sweep's reads past the values stay inside)
__host__ __device__ __forceinline__ size_t round16(size_t b) { return (b + 15) & ~(size_t)15; }

// entries of a block's window: its slices and its pivots
__host__ __device__ __forceinline__ size_t ilu_window(size_t nr, size_t dp) { return 32 * dp + ((nr + 31) & ~(size_t)31); }

// u16 words of a block's record: first slice of each level of the lower
// (nl + 1) and of the upper sweep (nu + 1), the slices' starts / 32 (lower,
// upper, end), then the rows of the lower and of the upper slices' lanes
// (kIluNoRow past a level's last), padded to 16 bytes
constexpr unsigned short kIluNoRow = 0xffff;
__host__ __device__ __forceinline__ size_t ilu_meta_words(size_t nl, size_t nu, size_t nsl, size_t nsu) {
    return (nl + nu + 3 + 33 * (nsl + nsu) + 7) & ~(size_t)7;
}

// entries that a sweep may read past the last slice: values of any kind, columns
// of zero (a place of the vector); part of each block's columns and window
constexpr int kIluSlack = 256;
__host__ __device__ __forceinline__ size_t ilu_columns(size_t dp) { return 32 * dp + kIluSlack; }

// shared bytes of the staged kernels for one block (host and device agree)
__host__ __device__ __forceinline__ size_t ilu_stage_bytes(size_t nr, size_t dp, size_t mw, size_t sz) {
    return round16((nr + 1) * sz) + ilu_window(nr, dp) * sz + ilu_columns(dp) * 2 + 2 * mw + 16 + kIluSlack * sz;
}

// The dynamic shared memory of the sweeps' kernels; the block's vector is at
// its start.  The staged factor is addressed by offsets from it, so that every
// access is known to be one to shared memory.
__device__ __forceinline__ unsigned char* ilu_smem() {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    return smem_raw;
}
// a block's factor and record for the sweeps, staged in shared memory ...
template <class T> struct IluShared {
    unsigned ov, oc, om;   // offsets of the values, the columns and the record
    int nl, nu, nsl, nsu, dp;
    __device__ __forceinline__ unsigned meta(int i) const {
        return *reinterpret_cast<const unsigned short*>(ilu_smem() + om + 2 * i);
    }
    __device__ __forceinline__ T val(int i) const { return reinterpret_cast<const T*>(ilu_smem() + ov)[i]; }
    __device__ __forceinline__ unsigned col(int i) const {
        return reinterpret_cast<const unsigned short*>(ilu_smem() + oc)[i];
    }
};
// ... or read in place
template <class T> struct IluGlobal {
    const T* v;
    const unsigned short *c, *m;
    int nl, nu, nsl, nsu, dp;
    __device__ __forceinline__ unsigned meta(int i) const { return m[i]; }
    __device__ __forceinline__ T val(int i) const { return v[i]; }
    __device__ __forceinline__ unsigned col(int i) const { return c[i]; }
};
template <class V, class A, class C, class M> __device__ __forceinline__ V ilu_view(const IluBlk& B, A v, C c, M m) {
    return V{v, c, m, B.nl, B.nu, B.nsl, B.nsu, B.dp};
}
// the record's parts (ilu_meta_words)
template <class V> __device__ __forceinline__ int ilu_level(const V& f, bool upper, int l) {
    return (int)f.meta((upper ? f.nl + 1 : 0) + l);
}
template <class V> __device__ __forceinline__ int ilu_start(const V& f, bool upper, int s) {
    return (int)f.meta(f.nl + f.nu + 2 + (upper ? f.nsl : 0) + s);
}
template <class V> __device__ __forceinline__ int ilu_row(const V& f, bool upper, int q) {
    return (int)f.meta(f.nl + f.nu + 3 + f.nsl + f.nsu + (upper ? 32 * f.nsl : 0) + q);
}

// a staged block: where its parts sit in shared memory
template <class T> struct IluStage {
    T* x;
    T* val;
    unsigned short* col;
    unsigned short* meta;
    uint64_t* bar;
    unsigned ov, oc, om;
    __device__ __forceinline__ IluStage(const IluBlk& B, int nr) {
        unsigned char* smem = ilu_smem();
        ov = (unsigned)round16(sizeof(T) * (nr + 1));
        oc = ov + (unsigned)(sizeof(T) * ilu_window(nr, B.dp));
        om = oc + 2u * (unsigned)ilu_columns(B.dp);
        x = reinterpret_cast<T*>(smem);
        val = reinterpret_cast<T*>(smem + ov);
        col = reinterpret_cast<unsigned short*>(smem + oc);
        meta = reinterpret_cast<unsigned short*>(smem + om);
        bar = reinterpret_cast<uint64_t*>(smem + om + 2u * B.mw);
    }
    __device__ __forceinline__ IluShared<T> view(const IluBlk& B) const {
        return ilu_view<IluShared<T>>(B, ov, oc, om);
    }
};

// the copies of a block's values (lu), columns and record, by one thread; the
// barrier has been initialised with a count of one
template <class T>
__device__ __forceinline__ void ilu_stage_bulk(const IluStage<T>& S, const IluBlk& B, int nr, const T* lu,
                                               const unsigned short* lu_col, const unsigned short* meta) {
    if (threadIdx.x == 0) {
        const uint32_t b = tc05::smem_u32(S.bar);
        const uint32_t vb = (uint32_t)(ilu_window(nr, B.dp) * sizeof(T)), cb = 2u * (uint32_t)ilu_columns(B.dp), mb = 2u * (uint32_t)B.mw;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(vb + cb + mb) : "memory");
        tc05::bulk_g2s(S.val, lu + B.v0, vb, S.bar);
        tc05::bulk_g2s(S.col, lu_col + B.c0, cb, S.bar);
        tc05::bulk_g2s(S.meta, meta + B.mo, mb, S.bar);
    }
}

// The thread's index, read anew: what follows from it is computed where it is
// used.  Kept across the other phases of a persistent kernel that needs all
// its registers for them, it would be spilled, and its L1 lines evicted by what
// those phases stream.
__device__ __forceinline__ int tid_here() {
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}

// One triangular sweep over the levels [l0, l1): rows of a level are
// independent, a warp takes a slice of 32.  UPPER: x_i = (x_i - sum over the
// upper entries) * inverse pivot; else x_i = x_i - sum over the lower ones
// (unit lower triangle).  A warp's slice of level l+1 -- its rows and the first
// kIluPre columns, which do not depend on x -- is fetched while level l is
// computed, so after each barrier only the x loads (independent of each other,
// the values loaded beside them) and the accumulation remain on the critical
// path; a warp without a slice goes straight to the barrier.  Entries in column
// order.  All bounds are the same for a warp's lanes; loads are taken four
// entries at a time, past a slice's last entry (kIluSlack entries after the
// arrays), and what lies there is left unused.
// Most rows of a tetrahedral mesh have more than kIluPre entries (up to 14), but
// a level is bound by the instructions that its warps issue: the two sweeps of
// a 1,447-row block of the 214k-node box took 5.0 us with 4 columns fetched
// ahead, 5.1 with 8 and more with 12 and 16.  Stored row by row with a row per
// lane they took 9.2 us.
constexpr int kIluPre = 4;
struct IluLane {
    int row, w, at;
    unsigned c[kIluPre];
};

template <bool UPPER, class V>
__device__ __forceinline__ void ilu_fetch(IluLane& R, const V& f, int lane, int s) {
    const int p = ilu_start(f, UPPER, s);
    R.w = ilu_start(f, UPPER, s + 1) - p;
    R.at = 32 * p + lane;
    R.row = ilu_row(f, UPPER, 32 * s + lane);
#pragma unroll
    for (int k = 0; k < kIluPre; ++k) R.c[k] = f.col(R.at + 32 * k);
}

// acc += entries [k, w) of a row
template <class T, class V>
__device__ __forceinline__ void ilu_rest(T& acc, const T* x, const V& f, int at, int w, int k) {
#pragma unroll 1
    for (; k < w; k += 4) {
        T v[4], xv[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            xv[t] = x[f.col(at + 32 * (k + t))];
            v[t] = f.val(at + 32 * (k + t));
        }
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (k + t < w) acc += v[t] * xv[t];
    }
}

template <class T, bool UPPER, class V>
__device__ __forceinline__ void ilu_sweep(const V& f, int l0, int l1) {
    T* const x = reinterpret_cast<T*>(ilu_smem());
    const int tid = tid_here(), warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
    // set before the conditional fetches: registers that a loop writes only
    // under a condition count as live all the way round it
    IluLane cur, nxt;
    cur.row = kIluNoRow;
    cur.w = cur.at = 0;
#pragma unroll
    for (int k = 0; k < kIluPre; ++k) cur.c[k] = 0;
    nxt = cur;
    if (l0 >= l1) return;
    int s0 = ilu_level(f, UPPER, l0), s1 = ilu_level(f, UPPER, l0 + 1);
    if (s0 + warp < s1) ilu_fetch<UPPER>(cur, f, lane, s0 + warp);
#pragma unroll 1
    for (int l = l0; l < l1; ++l) {
        const int s2 = l + 1 < l1 ? ilu_level(f, UPPER, l + 2) : s1;
        const bool more = s1 + warp < s2;
        if (s0 + warp < s1) {
            // this level's x and value loads first, then the next level's
            // slice while they are in flight, then the accumulation
            T xv[kIluPre], v[kIluPre];
#pragma unroll
            for (int k = 0; k < kIluPre; ++k) {
                xv[k] = x[cur.c[k]];
                v[k] = f.val(cur.at + 32 * k);
            }
            const bool act = cur.row != kIluNoRow;
            const int row = act ? cur.row : 0;
            const T xi = x[row], piv = UPPER ? f.val(32 * f.dp + row) : (T)1;
            if (more) ilu_fetch<UPPER>(nxt, f, lane, s1 + warp);
            T acc = (T)0;
#pragma unroll
            for (int k = 0; k < kIluPre; ++k)
                if (k < cur.w) acc += v[k] * xv[k];
            ilu_rest(acc, x, f, cur.at, cur.w, kIluPre);
            if (act) x[row] = UPPER ? (xi - acc) * piv : xi - acc;
            // slices of a level with more of them than the CTA has warps
#pragma unroll 1
            for (int s = s0 + warp + nw; s < s1; s += nw) {
                const int p = ilu_start(f, UPPER, s), w = ilu_start(f, UPPER, s + 1) - p;
                const int i = ilu_row(f, UPPER, 32 * s + lane);
                T a = (T)0;
                ilu_rest(a, x, f, 32 * p + lane, w, 0);
                if (i != kIluNoRow) x[i] = UPPER ? (x[i] - a) * f.val(32 * f.dp + i) : x[i] - a;
            }
        } else if (more) {
            ilu_fetch<UPPER>(nxt, f, lane, s1 + warp);
        }
        __syncthreads();
        cur = nxt;
        s0 = s1;
        s1 = s2;
    }
}

} // namespace fvmb
