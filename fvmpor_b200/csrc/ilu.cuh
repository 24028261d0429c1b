// Block-ILU(0) preconditioner state and the device helpers of its
// shared-memory ("staged") triangular solves, shared by the preconditioner
// kernels (precond.cu) and the fused Arnoldi kernel (arnoldi_fused.cu).
#pragma once

#include "ctx.cuh"
#include "ilu_layout.hpp"
#include "tc05.cuh"

#include <cstdint>
#include <vector>

namespace fvmb {

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
    bool wide = false;        // a block has wide rows
    // the set-up's Jacobian in factor order, for an FP64 and an FP32 factor
    // (written by the quotient kernels; allocated at the first use of each)
    DevBuf<double> Jw;
    DevBuf<float> Jw32;
    DevBuf<int> lu_up;        // [N] IluPlaces::upper (blocks not staged)
    DevBuf<int> lu_row;       // global row of each factor position (colour order inside the blocks)
    // ILU(0) elimination schedule of the shared-memory factorisation, one
    // contiguous segment per level (upd[seg_ptr[g] .. seg_ptr[g+1]), g the
    // block's first level (IluBlk::seg) plus the level): the offset of the
    // list of each lane of the level's groups, then per row and per L entry
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
    bool schur_staged[2] = {false, false};   // its factor in shared memory, or read in place
};

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
// Shared layout: x[T nr + 1, 16-B padded] | val[T wn] | col[u16 ds + slack] |
// record | mbarrier (a sweep's reads past the values stay inside)
// (sizes in ilu_layout.hpp)
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
    int nl, nu, ngl, ngu, nwide, ds;
    __device__ __forceinline__ unsigned meta(int i) const {
        return *reinterpret_cast<const unsigned short*>(ilu_smem() + om + 2 * i);
    }
    __device__ __forceinline__ unsigned meta2(int i) const {   // a double word, i even
        return *reinterpret_cast<const unsigned*>(ilu_smem() + om + 2 * i);
    }
    __device__ __forceinline__ T val(int i) const { return reinterpret_cast<const T*>(ilu_smem() + ov)[i]; }
    __device__ __forceinline__ unsigned col(int i) const {
        return reinterpret_cast<const unsigned short*>(ilu_smem() + oc)[i];
    }
    // the vector's value for a column; the padding's column is nr, a slot of its own
    static __device__ __forceinline__ T x(unsigned c) { return reinterpret_cast<const T*>(ilu_smem())[c]; }
};
// ... or read in place, where the vector may fill the shared memory to the last
// value and has no such slot
template <class T> struct IluGlobal {
    const T* v;
    const unsigned short *c, *m;
    int nl, nu, ngl, ngu, nwide, ds;
    unsigned nr;
    __device__ __forceinline__ T x(unsigned c) const { return c < nr ? reinterpret_cast<const T*>(ilu_smem())[c] : (T)0; }
    __device__ __forceinline__ unsigned meta(int i) const { return m[i]; }
    __device__ __forceinline__ unsigned meta2(int i) const { return *reinterpret_cast<const unsigned*>(m + i); }
    __device__ __forceinline__ T val(int i) const { return v[i]; }
    __device__ __forceinline__ unsigned col(int i) const { return c[i]; }
};
template <class T>
__device__ __forceinline__ IluGlobal<T> ilu_in_place(const IluBlk& B, int nr, const T* v, const unsigned short* c,
                                                     const unsigned short* m) {
    return IluGlobal<T>{v + B.v0, c + B.c0, m + B.mo, B.nl, B.nu, B.ngl, B.ngu, B.nwide, B.ds, (unsigned)nr};
}
// the record's parts (ilu_meta_words); g counts a sweep's groups from 0
template <class V> __device__ __forceinline__ int ilu_level(const V& f, bool upper, int l) {
    return (int)f.meta((upper ? f.nl + 1 : 0) + l);
}
template <class V> __device__ __forceinline__ int ilu_groups_at(const V& f) { return (f.nl + f.nu + 3) & ~1; }
template <class V> __device__ __forceinline__ int ilu_group_at(const V& f, bool upper, int g) {
    return ilu_groups_at(f) + 2 * ((upper ? f.ngl : 0) + g);
}
template <class V> __device__ __forceinline__ int ilu_row_at(const V& f, bool upper, int g, int j) {
    return ilu_groups_at(f) + 2 * (f.ngl + f.ngu + (int)kIluPad) + kIluGroup * ((upper ? f.ngl : 0) + g) + j;
}
template <class V> __device__ __forceinline__ int ilu_row(const V& f, bool upper, int g, int j) {
    return (int)f.meta(ilu_row_at(f, upper, g, j));
}
// a wide row's first entry past kIluWide and its entries, (0, 0) for a group that
// is none; only where the block has any (nwide)
template <class V> __device__ __forceinline__ int2 ilu_wide(const V& f, bool upper, int g) {
    const int at = ilu_groups_at(f) + (2 + kIluGroup) * (f.ngl + f.ngu + (int)kIluPad), key = (upper ? f.ngl : 0) + g;
    int lo = 0;
    for (int n = f.nwide; n > 1;) {   // ascending groups
        const int h = n >> 1;
        if ((int)f.meta2(at + 6 * (lo + h)) <= key) lo += h;
        n -= h;
    }
    if ((int)f.meta2(at + 6 * lo) != key) return make_int2(0, 0);
    return make_int2((int)f.meta2(at + 6 * lo + 2), (int)f.meta2(at + 6 * lo + 4));
}
// where the entries of lane j's row of a group are: the general form, for the
// factorisations
struct IluSpan {
    int at, tail, w;
    __device__ __forceinline__ int entry(int k) const { return k < kIluWide ? at + 32 * k : tail + k - kIluWide; }
};
template <class V> __device__ __forceinline__ IluSpan ilu_span(const V& f, bool upper, int g, int j) {
    const unsigned word = f.meta2(ilu_group_at(f, upper, g));
    IluSpan s{(int)(word >> kIluWidthBits) + j, 0, (int)(word & ((1u << kIluWidthBits) - 1u))};
    if (f.nwide) {
        const int2 t = ilu_wide(f, upper, g);
        if (t.y) {
            s.tail = t.x;
            s.w = t.y;
        }
    }
    return s;
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
        oc = ov + (unsigned)(sizeof(T) * ilu_window(nr, B.ds));
        om = oc + 2u * (unsigned)ilu_columns(B.ds);
        x = reinterpret_cast<T*>(smem);
        val = reinterpret_cast<T*>(smem + ov);
        col = reinterpret_cast<unsigned short*>(smem + oc);
        meta = reinterpret_cast<unsigned short*>(smem + om);
        bar = reinterpret_cast<uint64_t*>(smem + om + 2u * B.mw);
    }
    __device__ __forceinline__ IluShared<T> view(const IluBlk& B) const {
        return IluShared<T>{ov, oc, om, B.nl, B.nu, B.ngl, B.ngu, B.nwide, B.ds};
    }
};

// the copies of a block's values (lu), columns and record, by one thread; the
// barrier has been initialised with a count of one
template <class T>
__device__ __forceinline__ void ilu_stage_bulk(const IluStage<T>& S, const IluBlk& B, int nr, const T* lu,
                                               const unsigned short* lu_col, const unsigned short* meta) {
    if (threadIdx.x == 0) {
        const uint32_t b = tc05::smem_u32(S.bar);
        const uint32_t vb = (uint32_t)(ilu_window(nr, B.ds) * sizeof(T)), cb = 2u * (uint32_t)ilu_columns(B.ds), mb = 2u * (uint32_t)B.mw;
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
// independent, a warp takes a slice of kIluSlice groups.  UPPER: x_i = (x_i - sum
// over the upper entries) * inverse pivot; else x_i = x_i - sum over the lower
// ones (unit lower triangle).  A warp's slice of level l+1 -- its rows and the
// first kIluPre columns, which do not depend on x -- is fetched while level l is
// computed, so after each barrier only the x loads (independent of each other,
// the values loaded beside them) and the accumulation remain on the critical
// path; a warp without a slice goes straight to the barrier.  Entries in column
// order.  Loads are taken four entries at a time, past a group's last entry
// (kIluSlack entries after the arrays), and what lies there is left unused, as
// is what the lanes past a level's last group read (the next groups' entries).
// Most rows of a tetrahedral mesh have more than kIluPre entries (up to 14), but
// a level is bound by the instructions that its warps issue (so wide rows, WIDE,
// have a form of their own: with their code in every level an apply on the
// 214k-node box took 12.7 us instead of 12.2): the two sweeps of
// a 1,447-row block of the 214k-node box took 5.0 us with 4 columns fetched
// ahead, 5.1 with 8 and more with 12 and 16 (with slices of 32 rows).  Stored row
// by row with a row per lane they took 9.2 us.  One common bound for a slice's lanes
// in the loop over the rest, so that they do not part, was slower (30-day run of
// that box: fused cycle 0.630 ms instead of 0.611).
constexpr int kIluPre = 4;
struct IluLane {
    int row, w, at;
    unsigned c[kIluPre];
};

// the lane's row of a slice from group s on, in a level that ends at g1 (past it:
// no row); gw, gr: places of its group's word and of its row there for s = 0
template <class V>
__device__ __forceinline__ void ilu_fetch(IluLane& R, const V& f, int gw, int gr, int j, bool in, int s) {
    const unsigned word = f.meta2(gw + 2 * s);
    const int row = (int)f.meta(gr + kIluGroup * s);
    R.w = in ? (int)(word & ((1u << kIluWidthBits) - 1u)) : 0;
    R.at = (int)(word >> kIluWidthBits) + j;
    R.row = in ? row : kIluNoRow;
#pragma unroll
    for (int k = 0; k < kIluPre; ++k) R.c[k] = f.col(R.at + 32 * k);
}

// acc += entries [k, w) of a row in the strip
template <class T, class V>
__device__ __forceinline__ void ilu_rest(T& acc, const V& f, int at, int w, int k) {
#pragma unroll 1
    for (; k < w; k += 4) {
        T v[4], xv[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const unsigned c = f.col(at + 32 * (k + t));
            xv[t] = f.x(c);
            v[t] = f.val(at + 32 * (k + t));
        }
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (k + t < w) acc += v[t] * xv[t];
    }
}
// ... and a wide row's others
template <class T, class V> __device__ __forceinline__ T ilu_wide_rest(T acc, const V& f, bool upper, int g) {
    const int2 t = ilu_wide(f, upper, g);
#pragma unroll 1
    for (int k = 0; k < t.y - kIluWide; ++k) acc += f.val(t.x + k) * f.x(f.col(t.x + k));
    return acc;
}

template <class T, bool UPPER, bool WIDE, class V>
__device__ __forceinline__ void ilu_sweep(const V& f, int l0, int l1) {
    T* const x = reinterpret_cast<T*>(ilu_smem());
    const int tid = tid_here(), stride = (blockDim.x >> 5) * kIluSlice;
    const int first = (tid >> 5) * kIluSlice, mine = tid / kIluGroup;   // the warp's and the lane's group of a level
    const int j = tid & (kIluGroup - 1), gw = ilu_group_at(f, UPPER, mine), gr = ilu_row_at(f, UPPER, mine, j);
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
    if (s0 + first < s1) ilu_fetch(cur, f, gw, gr, j, s0 + mine < s1, s0);
#pragma unroll 1
    for (int l = l0; l < l1; ++l) {
        const int s2 = l + 1 < l1 ? ilu_level(f, UPPER, l + 2) : s1;
        const bool more = s1 + first < s2;
        if (s0 + first < s1) {
            // this level's x and value loads first, then the next level's
            // slice while they are in flight, then the accumulation
            T xv[kIluPre], v[kIluPre];
#pragma unroll
            for (int k = 0; k < kIluPre; ++k) {
                xv[k] = f.x(cur.c[k]);
                v[k] = f.val(cur.at + 32 * k);
            }
            const bool act = cur.row != kIluNoRow;
            const int row = act ? cur.row : 0;
            const T xi = x[row], piv = UPPER ? f.val(f.ds + row) : (T)1;
            if (more) ilu_fetch(nxt, f, gw, gr, j, s1 + mine < s2, s1);
            T acc = (T)0;
#pragma unroll
            for (int k = 0; k < kIluPre; ++k)
                if (k < cur.w) acc += v[k] * xv[k];
            ilu_rest(acc, f, cur.at, cur.w, kIluPre);
            if (WIDE && act) acc = ilu_wide_rest(acc, f, UPPER, s0 + mine);
            if (act) x[row] = UPPER ? (xi - acc) * piv : xi - acc;
            // slices of a level with more of them than the CTA has warps
#pragma unroll 1
            for (int s = s0 + stride; s + first < s1; s += stride) {
                const unsigned word = f.meta2(gw + 2 * s);
                const int i = s + mine < s1 ? (int)f.meta(gr + kIluGroup * s) : kIluNoRow;
                T a = (T)0;
                if (i != kIluNoRow) {
                    ilu_rest(a, f, (int)(word >> kIluWidthBits) + j, (int)(word & ((1u << kIluWidthBits) - 1u)), 0);
                    if (WIDE) a = ilu_wide_rest(a, f, UPPER, s + mine);
                    x[i] = UPPER ? (x[i] - a) * f.val(f.ds + i) : x[i] - a;
                }
            }
        } else if (more) {
            ilu_fetch(nxt, f, gw, gr, j, s1 + mine < s2, s1);
        }
        __syncthreads();
        cur = nxt;
        s0 = s1;
        s1 = s2;
    }
}

// for kernels that take both kinds of block
template <class T, bool UPPER, class V> __device__ __forceinline__ void ilu_sweep_any(const V& f, int l0, int l1) {
    if (f.nwide) ilu_sweep<T, UPPER, true>(f, l0, l1);
    else ilu_sweep<T, UPPER, false>(f, l0, l1);
}

} // namespace fvmb
