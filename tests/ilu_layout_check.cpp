// Walks the factor layout of ilu_layout.hpp on the host exactly as the device
// sweeps do (ilu.cuh: lanes past a level's last group, reads past a group's
// last entry) and compares with a row-by-row solve.  Arguments: rows, entries
// per row, rows of many entries, their entries, seed.  Prints the window's
// entries over the factor's own.
#include "ilu_layout.hpp"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <set>

using namespace fvmb;

#define CHECK(cond)                                                     \
    do {                                                                \
        if (!(cond)) { std::printf("line %d: %s\n", __LINE__, #cond); return 1; } \
    } while (0)

int main(int argc, char** argv) {
    if (argc != 6) return 2;
    const int nr = std::atoi(argv[1]), per_row = std::atoi(argv[2]), hubs = std::atoi(argv[3]);
    const int hub_len = std::atoi(argv[4]), r0 = 3;   // (a block need not start at row 0)
    std::mt19937 rng(std::atoi(argv[5]));
    // a block read in place may fill a CTA's shared memory to the last value
    CHECK(ilu_plain_bytes(29056, 8) <= kMaxDynSmem && ilu_plain_bytes(58112, 4) <= kMaxDynSmem);
    std::vector<std::set<int>> adj(nr);
    auto couple = [&](int a, int b) { adj[a].insert(b); adj[b].insert(a); };
    for (int i = 0; i < nr; ++i) {
        adj[i].insert(i);
        for (int k = 0; k < per_row / 2; ++k) couple(i, (int)(rng() % nr));
    }
    for (int h = 0; h < hubs; ++h)
        for (int i = (int)(rng() % nr), k = 0; k < hub_len; ++k) couple(i, (int)(rng() % nr));
    std::vector<int> ptr(r0 + nr + 1, 0), diag(r0 + nr);
    std::vector<unsigned short> col;
    for (int i = 0; i < nr; ++i) {
        for (int j : adj[i]) {
            if (j == i) diag[r0 + i] = (int)col.size();
            col.push_back((unsigned short)j);
        }
        ptr[r0 + i + 1] = (int)col.size();
    }
    // levels of the two sweeps
    std::vector<int> lptr(1, r0), lrows, uptr(1, r0), urows;
    int n_levels[2] = {0, 0};
    for (int up = 0; up < 2; ++up) {
        std::vector<int> lvl(nr, 0);
        int n = 0;
        for (int k = 0; k < nr; ++k) {
            const int i = up ? nr - 1 - k : k;
            for (int j : adj[i])
                if (up ? j > i : j < i) lvl[i] = std::max(lvl[i], lvl[j] + 1);
            n = std::max(n, lvl[i] + 1);
        }
        std::vector<int>&rows = up ? urows : lrows, &p = up ? uptr : lptr;
        rows.assign(r0, -1);
        for (int l = 0; l < n; ++l) {
            for (int i = 0; i < nr; ++i)
                if (lvl[i] == l) rows.push_back(r0 + i);
            p.push_back((int)rows.size());
        }
        n_levels[up] = n;
    }
    IluPlaces place;
    place.entry.assign(col.size(), -1);
    place.upper.assign(r0 + nr, -1);
    place.lower.assign(r0 + nr, -1);
    std::vector<unsigned short> meta, cols;
    const IluBlk B = ilu_layout(r0, r0 + nr, ptr, diag, col, {lptr, lrows, 0, n_levels[0]}, {uptr, urows, 0, n_levels[1]},
                                place, meta, cols);
    const size_t window = ilu_window(nr, B.ds);
    CHECK(cols.size() == ilu_columns(B.ds) && cols.size() % 8 == 0 && window % 4 == 0);
    CHECK((int)meta.size() == B.mw && meta.size() % 8 == 0);
    // every entry has a place of its own
    std::vector<double> val(window, 0.0);
    std::vector<char> taken(window, 0);
    std::vector<double> a(col.size());
    for (size_t e = 0; e < col.size(); ++e) {
        const int w = place.entry[e];
        CHECK(w >= 0 && (size_t)w < window && !taken[w]);
        taken[w] = 1;
        val[w] = a[e] = 0.1 + (double)(rng() % 1000) / 1000.0;
    }
    for (unsigned short c : cols) CHECK(c <= nr);
    // values behind the window that a sweep may read: of any kind
    val.resize(window + ilu_columns(B.ds), NAN);
    std::vector<double> x(nr + 1, 0.0), y(nr);
    for (int i = 0; i < nr; ++i) x[i] = y[i] = (double)(rng() % 2000) / 1000.0 - 1.0;
    auto meta2 = [&](int i) { return (unsigned)meta[i] | (unsigned)meta[i + 1] << 16; };
    const int at0 = (B.nl + B.nu + 3) & ~1, ng = B.ngl + B.ngu, rows0 = at0 + 2 * (ng + (int)kIluPad);
    const int wide0 = rows0 + kIluGroup * (ng + (int)kIluPad);
    CHECK(wide0 + 6 * B.nwide <= (int)meta.size());
    const int reach = B.ds + kIluSlack;   // ilu_stage_bytes
    for (int up = 0; up < 2; ++up) {
        const int n = n_levels[up], gbase = up ? B.ngl : 0;
        for (int l = 0; l < n; ++l) {
            const int g0 = meta[(up ? B.nl + 1 : 0) + l], g1 = meta[(up ? B.nl + 1 : 0) + l + 1];
            CHECK(g0 < g1 && g1 <= (up ? B.ngu : B.ngl));
            for (int s = g0; s < g1; s += kIluSlice) {
                std::set<int> columns, pairs[2];
                for (int lane = 0; lane < 32; ++lane) {
                    const int g = s + lane / kIluGroup, j = lane % kIluGroup;
                    const int word_at = at0 + 2 * (gbase + g), row_at = rows0 + kIluGroup * (gbase + g) + j;
                    CHECK(word_at + 1 < rows0 && row_at < wide0);
                    const unsigned word = meta2(word_at);
                    const int at = (int)(word >> kIluWidthBits) + j;
                    const int w = g < g1 ? (int)(word & ((1u << kIluWidthBits) - 1u)) : 0;
                    const int row = g < g1 ? meta[row_at] : kIluNoRow;
                    CHECK(w <= kIluWide);
                    if (g < g1 && j == 0 && w > 0) {
                        CHECK(columns.insert(at % 32 / kIluGroup).second);
                        CHECK(pairs[lane / 16].insert(at % 16 / kIluGroup).second);
                    }
                    double acc = 0.0;
                    for (int k = 0; k < std::max(4, (w + 3) & ~3); ++k) {
                        CHECK(at + 32 * k < reach);
                        const double v = val[at + 32 * k], xv = x[cols[at + 32 * k]];
                        if (k < w) acc += v * xv;
                    }
                    if (row == kIluNoRow) continue;
                    int t = 0;
                    while (t < B.nwide && (int)meta2(wide0 + 6 * t) != gbase + g) ++t;
                    if (t < B.nwide) {
                        CHECK(j == 0 && w == kIluWide);
                        const int tail = (int)meta2(wide0 + 6 * t + 2), len = (int)meta2(wide0 + 6 * t + 4);
                        for (int k = 0; k < len - kIluWide; ++k) acc += val[tail + k] * x[cols[tail + k]];
                    }
                    // the places of the factorisation's lists
                    if (up) CHECK(place.upper[r0 + row] == kIluGroup * g + j);
                    else CHECK(place.lower[r0 + row] == kIluGroup * (g - g0) + j);
                    x[row] = up ? (x[row] - acc) * val[B.ds + row] : x[row] - acc;
                }
            }
        }
        for (int k = 0; k < nr; ++k) {
            const int i = up ? nr - 1 - k : k;
            double acc = 0.0;
            for (int e = ptr[r0 + i]; e < ptr[r0 + i + 1]; ++e)
                if (up ? col[e] > i : col[e] < i) acc += a[e] * y[col[e]];
            y[i] = up ? (y[i] - acc) * a[diag[r0 + i]] : y[i] - acc;
        }
        for (int i = 0; i < nr; ++i) CHECK(x[i] == y[i] || std::fabs(x[i] - y[i]) <= 1e-12 * (std::fabs(y[i]) + 1.0));
        CHECK(x[nr] == 0.0);
    }
    std::printf("%.4f\n", (double)window / (double)col.size());
    return 0;
}
