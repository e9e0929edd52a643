// Host side of the grouped design's cell ranges (plain C++).
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace devil {

// The cells in key order (key = design row u * C + cluster) cut into slices of at
// most slice_cells cells of one design row, and, with clusters, into the pieces
// (slice x cluster) that the clustered bread/meat walks.
struct SliceCut {
    std::vector<int32_t> sl_start{0};  // [S + 1] first cell of every slice
    std::vector<int32_t> sl_key;       // [S] its design row
    std::vector<int32_t> kslice;       // [U + 1] first slice of every design row
    // C > 1: the pieces, ordered by key
    std::vector<int32_t> f_key;     // [NF] key
    std::vector<int32_t> f_slice;   // [NF] its slice
    std::vector<int32_t> f_base;    // [NF] first cell of its slice
    std::vector<int32_t> f_loc;     // [NF] its first cell, counted in the slice
    std::vector<int32_t> f_kslice;  // [U * C + 1] first piece of every key
    bool by_cluster = false;        // the slices end at the clusters: every piece is a whole slice
};

// kst[U * C + 1]: first cell of every key
inline SliceCut cut_slices(const std::vector<int64_t>& kst, int U, int C, int slice_cells, bool by_cluster) {
    SliceCut cut;
    cut.by_cluster = by_cluster || C == 1;
    cut.kslice.resize(U + 1);
    const int step = by_cluster ? 1 : C;
    for (int u = 0; u < U; ++u) {
        cut.kslice[u] = (int32_t)cut.sl_key.size();
        for (int k = u * C; k < (u + 1) * C; k += step) {
            const int64_t a = kst[k], cnt = kst[k + step] - a;
            const int64_t ranges = (cnt + slice_cells - 1) / slice_cells;
            for (int64_t q = 1; q <= ranges; ++q) {
                cut.sl_start.push_back((int32_t)(a + cnt * q / ranges));
                cut.sl_key.push_back(u);
            }
        }
    }
    cut.kslice[U] = (int32_t)cut.sl_key.size();
    if (C == 1) return cut;
    cut.f_kslice.resize((size_t)U * C + 1);
    int sl = 0;
    for (int k = 0; k < U * C; ++k) {
        cut.f_kslice[k] = (int32_t)cut.f_key.size();
        for (int64_t a = kst[k]; a < kst[k + 1];) {
            while (cut.sl_start[sl + 1] <= a) ++sl;  // (no slice is empty)
            cut.f_key.push_back(k);
            cut.f_slice.push_back(sl);
            cut.f_base.push_back(cut.sl_start[sl]);
            cut.f_loc.push_back((int32_t)(a - cut.sl_start[sl]));
            a = std::min<int64_t>(kst[k + 1], cut.sl_start[sl + 1]);
        }
    }
    cut.f_kslice[(size_t)U * C] = (int32_t)cut.f_key.size();
    return cut;
}

// The same, cut at the clusters where the pieces of slices that cross them are
// more than the clustered pass takes (fits(NF)): up to one piece per key and one
// per slice, against one per key and 16,384 cells.
template <class Fits>
SliceCut cut_slices_fitting(const std::vector<int64_t>& kst, int U, int C, int slice_cells, bool by_cluster,
                            Fits&& fits) {
    SliceCut cut = cut_slices(kst, U, C, slice_cells, by_cluster);
    if (!cut.by_cluster && !fits((int)cut.f_key.size())) cut = cut_slices(kst, U, C, slice_cells, true);
    return cut;
}

}  // namespace devil
