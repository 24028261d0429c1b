// Layout of a block's ILU(0) factor for the triangular sweeps: sizes shared with
// the kernels (ilu.cuh) and its construction on the host.
#pragma once

#include "common.hpp"
#include "cvfe_geom.cuh"

#include <algorithm>
#include <cstddef>
#include <vector>

namespace fvmb {

// One block's factor: rows in colour order, the off-diagonal entries arranged by
// level for the sweeps, a row per lane.  The rows of a level are taken longest
// first, kIluGroup to a group; a warp takes eight groups at a time.  A group's
// entries are four neighbouring lanes of a strip 32 lanes wide: entry k of its
// lane j at at + 32 k + j, at = 32 h + 4 c in the strip's column c, each row
// padded to the group's longest with zeros whose column is nr, a slot of the
// vector that stays zero.  The eight groups that a warp takes together sit in
// eight different columns, each column's groups stacked one under another, so
// a warp reads values and columns from 32 different banks (for FP64 values, its
// halves from 16 different pairs), and the addresses of a row's entries are one
// base and constants.  Stored row by row, with a row per lane, every read hit
// about four lanes' worth of bank conflicts, and the sweeps were bound by those.
// With slices of 32 rows padded to their longest, and to 32 rows at the end of
// each level, the window grew by 7 % on the 214k-node box in FP32 and doubled in
// the Schur order of small blocks (many short levels); in groups of four it is
// smaller than row by row there (120.4 KB against 124.4 and 133.1), and within
// 5 % of it in Schur order.
// A row of more than kIluWide entries on one side of the diagonal has a group
// to itself; its entries past kIluWide follow the strip, one after another.
// Then come the (inverted) pivots in row order.
constexpr int kIluGroup = 4;
constexpr int kIluSlice = 32 / kIluGroup;   // groups of a warp's lanes
constexpr int kIluWide = 64;
struct IluBlk {
    int v0;    // first entry in the value arrays (a multiple of 4)
    int c0;    // and in the column array (a multiple of 8)
    int ds;    // the pivots' first entry: strip and wide rows before it (a multiple of 8)
    int mo;    // the record's first word (a multiple of 8)
    int mw;    // its words
    int nl, nu;      // levels of the lower and the upper sweep
    int ngl, ngu;    // their groups
    int nwide;       // wide rows' groups
    int seg;     // first level in the elimination schedule
};

FVM_HD size_t round16(size_t b) { return (b + 15) & ~(size_t)15; }

// entries of a block's window: its strip, its wide rows' rests and its pivots
FVM_HD size_t ilu_window(size_t nr, size_t ds) { return ds + ((nr + 3) & ~(size_t)3); }

// u16 words of a block's record: first group of each level of the lower (nl + 1)
// and of the upper sweep (nu + 1); from an even word on, two words for each
// group, lower and upper (bits 7 and up: its at; below: its entries per row in
// the strip); the groups' rows (kIluNoRow for none); three double words for each
// wide row: group, first entry past kIluWide, entries; padded to 16 bytes.  A
// warp may read kIluSlice - 1 groups past the last one, words and rows.
constexpr unsigned short kIluNoRow = 0xffff;
constexpr unsigned kIluWidthBits = 7;
static_assert(kIluWide < 1 << kIluWidthBits, "the group's word");
constexpr size_t kIluPad = kIluSlice - 1;   // groups' words and rows behind the last
FVM_HD size_t ilu_meta_words(size_t nl, size_t nu, size_t ng, size_t nwide) {
    return (((nl + nu + 3) & ~(size_t)1) + (2 + kIluGroup) * (ng + kIluPad) + 6 * nwide + 7) & ~(size_t)7;
}

// entries that a sweep may read past the last one of the strip or the wide rows:
// values of any kind, columns of zero (a place of the vector); part of each
// block's columns
constexpr int kIluSlack = 128;
FVM_HD size_t ilu_columns(size_t ds) { return ds + kIluSlack; }

// shared bytes of the staged kernels for one block (host and device agree)
FVM_HD size_t ilu_stage_bytes(size_t nr, size_t ds, size_t mw, size_t sz) {
    const size_t x = round16((nr + 1) * sz), need = x + ilu_window(nr, ds) * sz + ilu_columns(ds) * 2 + 2 * mw + 16;
    const size_t reach = x + ilu_columns(ds) * sz;
    return need > reach ? need : round16(reach);
}

// shared bytes of a block's vector where the factor is read in place: no slot for
// the padding's column (IluGlobal::x)
FVM_HD size_t ilu_plain_bytes(size_t nr, size_t sz) { return nr * sz; }

// largest dynamic shared-memory carve-out a CTA may request on sm_100
constexpr size_t kMaxDynSmem = 227 * 1024;

// the levels of one sweep: block's are [first, last), level g's rows
// rows[ptr[g]] .. rows[ptr[g + 1] - 1]
struct IluLevels {
    const std::vector<int>& ptr;
    std::vector<int>& rows;
    int first, last;
};

// place of every entry in its block's window; of every row, its group * kIluGroup
// + its lane there in the upper sweep, and the same from its level's first
// group in the lower one
struct IluPlaces {
    std::vector<int> entry, upper, lower;
};

// Block [r0, r1) of the factor whose row i has the entries ptr[i] .. ptr[i + 1] - 1
// in column order (col: columns from r0, pivot at diag[i]): its layout (but for
// its first places in the arrays and its schedule), record and columns; orders
// each level's rows
inline IluBlk ilu_layout(int r0, int r1, const std::vector<int>& ptr, const std::vector<int>& diag,
                         const std::vector<unsigned short>& col, IluLevels lower, IluLevels upper, IluPlaces& place,
                         std::vector<unsigned short>& meta, std::vector<unsigned short>& cols) {
    IluBlk B{};
    B.nl = lower.last - lower.first;
    B.nu = upper.last - upper.first;
    struct Group {
        int row[kIluGroup] = {-1, -1, -1, -1};
        int w = 0, at = 0, tail = 0;
    };
    static_assert(kIluGroup == 4, "Group::row");
    std::vector<Group> groups;
    std::vector<int> first[2], slices;   // of each level; the groups that warps take together
    for (int up = 0; up < 2; ++up) {
        IluLevels& lv = up ? upper : lower;
        const int base = (int)groups.size();
        auto length = [&](int i) { return up ? ptr[i + 1] - diag[i] - 1 : diag[i] - ptr[i]; };
        first[up].push_back(0);
        for (int g = lv.first; g < lv.last; ++g) {
            // a level's rows longest first, stable
            std::stable_sort(lv.rows.begin() + lv.ptr[g], lv.rows.begin() + lv.ptr[g + 1],
                             [&](int x, int y) { return length(x) > length(y); });
            const int l0 = (int)groups.size();
            for (int q = lv.ptr[g]; q < lv.ptr[g + 1];) {
                Group k;
                k.w = length(lv.rows[q]);
                const int n = k.w > kIluWide ? 1 : std::min(kIluGroup, lv.ptr[g + 1] - q);
                for (int j = 0; j < n; ++j, ++q) {
                    const int i = k.row[j] = lv.rows[q];
                    if (up) place.upper[i] = kIluGroup * ((int)groups.size() - base) + j;
                    else place.lower[i] = kIluGroup * ((int)groups.size() - l0) + j;
                }
                groups.push_back(k);
            }
            for (int k = l0; k < (int)groups.size(); k += kIluSlice) slices.push_back(k);
            first[up].push_back((int)groups.size() - base);
        }
        (up ? B.ngu : B.ngl) = (int)groups.size() - base;
        slices.push_back((int)groups.size());   // where the last level's last slice ends
    }
    // Places in the strip: the tallest slices first, each slice's groups on the
    // columns of least height.  Columns c and c + 4 share banks of 8-byte
    // values, so a slice's first four groups take one of each such pair and its
    // last four the other.
    int height[kIluSlice] = {};
    auto strip_w = [&](int g) { return std::min(groups[g].w, kIluWide); };
    std::vector<int> order;
    for (size_t k = 0; k + 1 < slices.size(); ++k)
        if (slices[k] < slices[k + 1]) order.push_back((int)k);
    std::stable_sort(order.begin(), order.end(),
                     [&](int x, int y) { return strip_w(slices[x]) > strip_w(slices[y]); });
    constexpr int kHalf = kIluSlice / 2;
    for (int k : order) {
        int half[2][kHalf];
        for (int c = 0; c < kHalf; ++c) {
            half[0][c] = height[c] <= height[c + kHalf] ? c : c + kHalf;
            half[1][c] = 2 * c + kHalf - half[0][c];
        }
        for (auto& h : half) std::stable_sort(h, h + kHalf, [&](int x, int y) { return height[x] < height[y]; });
        const int n = slices[k + 1] - slices[k];
        for (int j = 0; j < n; ++j) {
            const int c = half[j / kHalf][j % kHalf];
            groups[slices[k] + j].at = 32 * height[c] + kIluGroup * c;
            height[c] += strip_w(slices[k] + j);
        }
    }
    long ds = 32l * *std::max_element(height, height + kIluSlice);
    for (Group& k : groups)
        if (k.w > kIluWide) {
            k.tail = (int)ds;
            ds += k.w - kIluWide;
            B.nwide++;
        }
    ds = (ds + 7) & ~7l;
    if (ds >= 1l << (32 - kIluWidthBits)) throw Error("block-ILU: block too large");
    B.ds = (int)ds;
    cols.assign(ds, (unsigned short)(r1 - r0));
    for (int g = 0; g < (int)groups.size(); ++g) {
        const Group& k = groups[g];
        for (int j = 0; j < kIluGroup; ++j) {
            const int i = k.row[j];
            if (i < 0) continue;
            const int e0 = g < B.ngl ? ptr[i] : diag[i] + 1, e1 = g < B.ngl ? diag[i] : ptr[i + 1];
            for (int e = e0; e < e1; ++e) {
                place.entry[e] = e - e0 < kIluWide ? k.at + 32 * (e - e0) + j : k.tail + e - e0 - kIluWide;
                cols[place.entry[e]] = col[e];
            }
        }
    }
    for (int i = r0; i < r1; ++i) place.entry[diag[i]] = B.ds + i - r0;
    cols.resize(ilu_columns(B.ds), 0);
    meta.clear();
    auto put2 = [&](unsigned v) {
        meta.push_back((unsigned short)(v & 0xffffu));
        meta.push_back((unsigned short)(v >> 16));
    };
    for (const std::vector<int>& v : first) meta.insert(meta.end(), v.begin(), v.end());
    if (meta.size() & 1) meta.push_back(0);
    for (const Group& k : groups) put2((unsigned)k.at << kIluWidthBits | (unsigned)std::min(k.w, kIluWide));
    meta.resize(meta.size() + 2 * kIluPad, 0);
    for (const Group& k : groups)
        for (int i : k.row) meta.push_back(i < 0 ? kIluNoRow : (unsigned short)(i - r0));
    meta.resize(meta.size() + kIluGroup * kIluPad, kIluNoRow);
    for (int g = 0; g < (int)groups.size(); ++g)
        if (groups[g].w > kIluWide) {
            put2((unsigned)g);
            put2((unsigned)groups[g].tail);
            put2((unsigned)groups[g].w);
        }
    meta.resize(ilu_meta_words(B.nl, B.nu, (size_t)B.ngl + B.ngu, B.nwide), 0);
    B.mw = (int)meta.size();
    return B;
}

} // namespace fvmb
