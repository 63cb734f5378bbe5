// Warp windows: 32 consecutive segments (vertices, with their exclusive
// degree prefix) held in a warp's registers, whose items (edges) the warp
// walks in rows of 32.  A lane finds the segment of its item with one ballot,
// one OR-reduction and a few shuffles; there is no CTA barrier, no shared
// memory and no per-item search, which is what bounds LbTile kernels whose
// work per item is one load and one store.
//
// A warp takes the merge-path tile [tile * T, (tile + 1) * T) of the sequence
// of items and segment ends (splits from lb_partition), so a run of empty
// segments costs as much as a run of items and every tile has bounded work.
#pragma once

#include "hn_internal.cuh"

namespace hn {

struct WarpTile {
    long long item0;   // first item
    int nitems;
    long long seg0;    // segment of the first item (or the first that ends here)
    long long seg1;    // last segment with items or an end in the tile
};

__device__ __forceinline__ WarpTile warp_tile(const long long* __restrict__ splits, long long tile,
                                              int T, long long total, long long nseg) {
    WarpTile w;
    const long long d1 = (tile + 1) * T < total + nseg ? (tile + 1) * T : total + nseg;
    const long long a0 = splits[tile], a1 = splits[tile + 1];
    w.item0 = a0;
    w.nitems = (int)(a1 - a0);
    w.seg0 = tile * T - a0;
    w.seg1 = d1 - a1 < nseg ? d1 - a1 : nseg - 1;
    return w;
}

// Lane k holds the k-th non-empty segment of the window.
struct WarpWindow {
    int start;         // its first item, relative to the tile's item0 (clamped to >= 0)
    int lane_of;       // the lane (segment s0 + lane_of) it came from
    int n;             // non-empty segments in the window
    int begin, end;    // the window's items, relative to item0
};

// The window of segments [s0, s0 + 32) of tile w.  `first` is the lane's
// prefix[s0 + lane] (any value past the tile's last segment).
__device__ __forceinline__ WarpWindow warp_window(const WarpTile& w, long long s0, long long first,
                                                  long long next_first) {
    const unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const bool in = s0 + lane <= w.seg1;
    const long long rel = first - w.item0;
    int st = !in ? w.nitems : rel < 0 ? 0 : (int)(rel < w.nitems ? rel : w.nitems);
    const long long nrel = next_first - w.item0;   // of segment s0 + 32
    const int wend = s0 + 32 > w.seg1 ? w.nitems : (int)(nrel < w.nitems ? nrel : w.nitems);
    int nx = __shfl_down_sync(kFull, st, 1);
    if (lane == 31) nx = wend;
    const unsigned full = __ballot_sync(kFull, in && nx > st);
    WarpWindow r;
    r.n = __popc(full);
    r.begin = __shfl_sync(kFull, st, 0);
    r.end = wend;
    // lane k: position of the k-th set bit of `full`
    int pos = 0;
    unsigned m = full;
    int k = lane;
#pragma unroll
    for (int h = 16; h; h >>= 1) {
        const int c = __popc(m & ((1u << h) - 1u));
        if (k >= c) {
            k -= c;
            pos += h;
            m >>= h;
        }
    }
    r.lane_of = pos & 31;
    st = __shfl_sync(kFull, st, r.lane_of);
    r.start = lane < r.n ? st : 0x7FFFFFFF;
    return r;
}

// The index (0..n-1) of the segment that holds item `row + lane` of the
// window; meaningless for lanes outside [begin, end).  Called by all lanes.
__device__ __forceinline__ int warp_owner(const WarpWindow& w, int row) {
    const unsigned kFull = 0xFFFFFFFFu;
    if (w.n == 1) return 0;
    const int lane = threadIdx.x & 31;
    const unsigned rel = (unsigned)(w.start - row);   // wraps for segments begun before the row
    const int before = __popc(__ballot_sync(kFull, w.start < row));
    const unsigned bits = __reduce_or_sync(kFull, rel < 32u ? 1u << rel : 0u);
    return before - 1 + __popc(bits & (kFull >> (31 - lane)));
}

}  // namespace hn
