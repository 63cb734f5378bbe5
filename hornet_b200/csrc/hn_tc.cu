// TriangleCounting2 (hornetsnest/src/Static/TriangleCounting/triangle2.cu:75-171
// with forAllAdjUnions, primitives/Operator++.i.cuh:319-522).
//
// The reference counts on a graph read with DIRECTED_BY_DEGREE | SORT
// (hornetsnest/test/TriangleTest2.cu:86-87): every undirected edge is kept
// once, from the lower-(degree, id) endpoint (xlib/src/Graph/GraphStd.cpp:
// 247-268), so each triangle is found exactly once.  It then bins all
// directed edges by log-degree pair with 64-bit global atomics (two passes)
// and runs ~37 intersection launches.
//
// Here the orientation is built on the device in two passes over the (always
// sorted) undirected adjacency: one decides every edge's direction and counts,
// one writes the kept neighbours (k_orient).  The intersection is
// vertex-centric (see the comment above k_tc_warp): N+(u) is a bitmap in shared
// memory, or a hash table where it spans too many numbers.
//
// Counts of graphs whose edges are not local in vertex id use numbers by
// descending rank in the (degree, id) order in place of ids, so that nearly
// all probes are among the first kWin numbers, a 16 KB bitmap.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "hn_graph.cuh"
#include "hn_tc.cuh"
#include "hn_window.cuh"

namespace hn {

namespace {

constexpr int kB = 256;
using Tile = LbTile<kB, 4>;

__device__ __forceinline__ bool oriented_before(int du, int u, int dv, int v) {
    return du < dv || (du == dv && u < v);
}

__global__ void __launch_bounds__(kB)
k_orient_flags(const long long* __restrict__ prefix, int nV, const VRec* __restrict__ vtab,
               const int32_t* __restrict__ pool, int32_t* __restrict__ flag,
               const long long* __restrict__ splits, long long split_tiles) {
    __shared__ Tile t;
    __shared__ long long s_base[Tile::TILE + 1];
    __shared__ int s_deg[Tile::TILE + 1];
    const long long total = prefix[nV];
    const long long ntiles = (total + nV + Tile::TILE - 1) / Tile::TILE;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        int n = lb_tile_load(t, prefix, (long long)nV, total, tile, splits, split_tiles);
        for (int b = threadIdx.x; b <= t.nends; b += kB) {
            long long u = t.seg0 + b;
            if (u < nV) {
                VRec r = vtab[u];
                s_base[b] = r.off - t.seg_start(b);
                s_deg[b] = r.deg;
            }
        }
        __syncthreads();
        // all of a thread's loads first: neighbours, then their degrees
        constexpr int IPT = Tile::TILE / kB;
        int bs[IPT], vs[IPT], dv[IPT];
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            const int i = threadIdx.x + k * kB;
            bs[k] = -1;
            if (i < n) {
                bs[k] = t.seg[i];
                vs[k] = pool[s_base[bs[k]] + t.item0 + i];
            }
        }
#pragma unroll
        for (int k = 0; k < IPT; k++)
            if (bs[k] >= 0) dv[k] = vtab[vs[k]].deg;
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            if (bs[k] < 0) continue;
            const int b = bs[k];
            const int u = (int)(t.seg0 + b);
            flag[t.item0 + threadIdx.x + k * kB] = oriented_before(s_deg[b], u, dv[k], vs[k]) ? 1 : 0;
        }
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) flag[total] = 0;
}

__global__ void __launch_bounds__(kB)
k_orient_fill(const long long* __restrict__ prefix, int nV, const VRec* __restrict__ vtab,
              const int32_t* __restrict__ pool, const int32_t* __restrict__ pos,
              int32_t* __restrict__ fwd, long long* __restrict__ offp,
              const long long* __restrict__ splits, long long split_tiles,
              const int32_t* __restrict__ canon, int32_t* __restrict__ feid) {
    __shared__ Tile t;
    __shared__ long long s_base[Tile::TILE + 1];
    const long long total = prefix[nV];
    const long long ntiles = (total + nV + Tile::TILE - 1) / Tile::TILE;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        int n = lb_tile_load(t, prefix, (long long)nV, total, tile, splits, split_tiles);
        for (int b = threadIdx.x; b <= t.nends; b += kB) {
            long long u = t.seg0 + b;
            if (u < nV) s_base[b] = vtab[u].off - t.seg_start(b);
        }
        __syncthreads();
        constexpr int IPT = Tile::TILE / kB;
        int ps[IPT], keep[IPT], vs[IPT];
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            const int i = threadIdx.x + k * kB;
            keep[k] = 0;
            if (i < n) {
                const long long e = t.item0 + i;
                ps[k] = pos[e];
                keep[k] = pos[e + 1] != ps[k];
                vs[k] = pool[s_base[t.seg[i]] + e];
            }
        }
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            if (!keep[k]) continue;
            const long long e = t.item0 + threadIdx.x + k * kB;
            fwd[ps[k]] = vs[k];
            if (feid) feid[ps[k]] = canon[e];   // edge id of the kept edge
        }
        __syncthreads();
    }
    // offp[u] = pos[prefix[u]]
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u <= nV;
         u += (long long)gridDim.x * blockDim.x)
        offp[u] = pos[prefix[u]];
}

// ---------------------------------------------------------------------------
// Orientation for counts.  A vertex's number is its id, or (ranked) its
// position in the descending (degree, id) order; its oriented list is stored
// under its number and holds numbers.  One 4-byte read per edge (the other
// end's degree or number; a vertex record is 16 bytes) decides the direction,
// kept as one bit per edge.  Lists are in the order of ids (not sorted by
// rank); each starts on 16 bytes and is padded to a multiple of four entries
// with kPad.
// ---------------------------------------------------------------------------
constexpr int kPad = INT_MAX;
constexpr int kWin = 1 << 17;   // numbers of the CTA kernel's bitmap (16 KB)
constexpr int kLocal = 1 << 17;  // ids closer than this are local
constexpr int kOrientTile = 1024;

__global__ void k_rank_keys(const VRec* __restrict__ vtab, int nV,
                            unsigned long long* __restrict__ keys) {
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < nV;
         v += (long long)gridDim.x * blockDim.x)
        keys[v] = ((unsigned long long)v << 32) | (unsigned)vtab[v].deg;
}

__global__ void k_rank_of(const unsigned long long* __restrict__ keys, int nV,
                          int32_t* __restrict__ rank, int32_t* __restrict__ inv) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nV;
         i += (long long)gridDim.x * blockDim.x) {
        const int v = (int)(keys[i] >> 32);
        rank[v] = nV - 1 - (int)i;
        inv[nV - 1 - i] = v;
    }
}

// Of evenly spaced edges, those whose ends are less than kLocal ids apart.
__global__ void k_local_sample(const long long* __restrict__ prefix, int nV, long long m,
                               const VRec* __restrict__ vtab, const int32_t* __restrict__ pool,
                               int samples, int* __restrict__ local) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool near = false;
    if (i < samples) {
        const long long e = (long long)((double)i / samples * m);
        const long long u = upper_bound_dev(prefix, (long long)nV + 1, e) - 1;
        const int v = pool[vtab[u].off + (e - prefix[u])];
        near = u - v < kLocal && v - u < kLocal;
    }
    const unsigned b = __ballot_sync(0xFFFFFFFFu, near);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(local, __popc(b));
}

__global__ void k_degree_of(const VRec* __restrict__ vtab, int nV, int32_t* __restrict__ deg) {
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < nV;
         v += (long long)gridDim.x * blockDim.x)
        deg[v] = vtab[v].deg;
}

// Bits of the row [row, row + 32) that belong to the lane's segment
// [w.start, send) of the window.
__device__ __forceinline__ unsigned own_bits(const WarpWindow& w, int send, int row) {
    const int lo = w.start > row ? w.start - row : 0;
    const int hi = send - row < 32 ? send - row : 32;
    if ((int)(threadIdx.x & 31) >= w.n || lo >= hi || hi <= 0 || lo > 31) return 0u;
    return (hi == 32 ? 0xFFFFFFFFu : (1u << hi) - 1u) & ~((1u << lo) - 1u);
}

// Pass 1 (FILL = false): the direction of every edge, one bit each in
// `kept`, the kept edges of each vertex in cnt[number], and those of each
// tile's last vertex in that tile in last[tile].  Pass 2 writes the numbers of
// the kept edges; a vertex that began in earlier tiles has their `last` edges
// before it.  key: numbers (RANKED) or degrees.  A warp per merge-path tile,
// windows of 32 vertices; a row of 32 edges is one word of `kept` (shared by
// two windows at their seam).
// R-MAT scale 22 (128 M edges): 1.26 ms both passes; the flags, scan and fill
// of build_oriented 3.4 ms (148 M edges in 512 graphs: 2.9 ms).
template <bool FILL, bool RANKED>
__global__ void __launch_bounds__(kB)
k_orient(const long long* __restrict__ prefix, int nV, long long nE,
         const VRec* __restrict__ vtab, const int32_t* __restrict__ pool,
         const int32_t* __restrict__ key, unsigned* __restrict__ kept,
         int* __restrict__ cnt, int* __restrict__ last, const long long* __restrict__ offp,
         int32_t* __restrict__ fwd, const long long* __restrict__ splits, long long ntiles) {
    constexpr int ROWS = 4;
    const unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const long long tile = blockIdx.x * (long long)(kB / 32) + (threadIdx.x >> 5);
    if (tile >= ntiles) return;
    const WarpTile wt = warp_tile(splits, tile, kOrientTile, nE, nV);
    if (wt.nitems == 0) return;
    int before = 0;   // kept edges of the tile's first vertex in earlier tiles
    if (FILL) {
        const long long p0 = prefix[wt.seg0];
        if (p0 < wt.item0) {
            for (long long j = (p0 + wt.seg0) / kOrientTile + lane; j < tile; j += 32)
                before += last[j];
            before = __reduce_add_sync(kFull, before);
        }
    }
    for (long long v0 = wt.seg0; v0 <= wt.seg1; v0 += 32) {
        const long long v = v0 + lane < nV ? v0 + lane : nV;
        const long long first = prefix[v];
        const long long next = v0 + 32 <= nV ? prefix[v0 + 32] : nE;
        const long long off = v < nV ? vtab[v].off : 0;
        const int kv = v < nV && (RANKED || !FILL) ? key[v] : 0;
        const WarpWindow w = warp_window(wt, v0, first, next);
        if (w.n == 0) continue;
        const long long base = __shfl_sync(kFull, off - first, w.lane_of) + wt.item0;
        const int ku = __shfl_sync(kFull, kv, w.lane_of);   // of the lane's segment
        const int id = (int)(v0 + w.lane_of);
        const int number = RANKED ? ku : id;
        // the lane's own segment [w.start, send)
        int send = __shfl_down_sync(kFull, w.start, 1);
        if (lane >= w.n - 1) send = w.end;
        const int row0 = w.begin - (int)((wt.item0 + w.begin) & 31);
        auto own = [&](int row) { return own_bits(w, send, row); };
        if (!FILL) {
            int mine = 0;
            for (int r = row0; r < w.end; r += 32 * ROWS) {
                int x[ROWS], u[ROWS], du[ROWS];
#pragma unroll
                for (int k = 0; k < ROWS; k++) {
                    const int row = r + 32 * k, e = row + lane;
                    x[k] = -1;
                    u[k] = du[k] = 0;
                    if (row < w.end) {   // uniform
                        const int j = warp_owner(w, row) & 31;
                        const long long b = __shfl_sync(kFull, base, j);
                        du[k] = __shfl_sync(kFull, ku, j);
                        if (!RANKED) u[k] = __shfl_sync(kFull, id, j);
                        if (e >= w.begin && e < w.end) x[k] = __ldcs(pool + b + e);
                    }
                }
#pragma unroll
                for (int k = 0; k < ROWS; k++) {
                    const int row = r + 32 * k;
                    if (row >= w.end) break;   // uniform
                    bool keep = false;
                    if (x[k] >= 0) {
                        const int kx = key[x[k]];
                        keep = RANKED ? kx < du[k] : oriented_before(du[k], u[k], kx, x[k]);
                    }
                    const unsigned b = __ballot_sync(kFull, keep);
                    mine += __popc(b & own(row));
                    if (lane == 0 && b) {
                        unsigned* word = kept + ((wt.item0 + row) >> 5);
                        if (row >= w.begin && row + 32 <= w.end) *word = b;
                        else atomicOr(word, b);
                    }
                }
            }
            if (lane < w.n && mine) atomicAdd(cnt + number, mine);
            if (lane < w.n && id == wt.seg1) last[tile] = mine;
        } else {
            // the next slot of the lane's segment
            long long at = 0;
            if (lane < w.n) at = offp[number] + (id == wt.seg0 ? before : 0);
            for (int r = row0; r < w.end; r += 32 * ROWS) {
                int x[ROWS];
                long long to[ROWS];
#pragma unroll
                for (int k = 0; k < ROWS; k++) {
                    const int row = r + 32 * k, e = row + lane;
                    x[k] = -1;
                    to[k] = 0;
                    if (row >= w.end) continue;   // uniform
                    const int j = warp_owner(w, row) & 31;
                    const unsigned b = kept[(wt.item0 + row) >> 5];
                    const unsigned seg = own(row);
                    const unsigned sj = __shfl_sync(kFull, seg, j);
                    const long long t0 = __shfl_sync(kFull, at, j);
                    const long long pb = __shfl_sync(kFull, base, j);
                    if (e >= w.begin && e < w.end && (b >> lane & 1u)) {
                        to[k] = t0 + __popc(b & sj & ((1u << lane) - 1u));
                        x[k] = __ldcs(pool + pb + e);
                    }
                    at += __popc(b & seg);
                }
#pragma unroll
                for (int k = 0; k < ROWS; k++)
                    if (x[k] >= 0) fwd[to[k]] = RANKED ? key[x[k]] : x[k];
            }
        }
    }
}

__global__ void k_max_int(const int* __restrict__ a, int n, int* __restrict__ out) {
    int mx = 0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        mx = max(mx, a[i]);
    mx = __reduce_max_sync(0xFFFFFFFFu, mx);
    if ((threadIdx.x & 31) == 0 && mx) atomicMax(out, mx);
}

__global__ void k_padded(const int* __restrict__ cnt, int nV, int* __restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i <= nV;
         i += (long long)gridDim.x * blockDim.x)
        out[i] = i < nV ? (cnt[i] + 3) & ~3 : 0;
}

__global__ void k_pad_lists(const long long* __restrict__ offp, const int* __restrict__ cnt,
                            int nV, int32_t* __restrict__ fwd) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nV;
         i += (long long)gridDim.x * blockDim.x)
        for (long long e = offp[i] + cnt[i]; e < offp[i + 1]; e++) fwd[e] = kPad;
}

// counts under numbers -> counts under vertex ids
__global__ void k_unrank(const unsigned long long* __restrict__ in,
                         const int32_t* __restrict__ inv, int nV,
                         unsigned long long* __restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nV;
         i += (long long)gridDim.x * blockDim.x)
        out[inv[i]] = in[i];
}

// Candidate lists.  The oriented edge x -> y contributes |N+(x) ∩ N+(y)|
// triangles whichever endpoint counts it, so it is counted by the endpoint
// whose out-list is the longer: that list is the hash table, the shorter
// one is probed (cost min(d+(x), d+(y)) instead of d+(y)).  C(z) lists the
// other endpoint of every edge z counts, stored as ~x when z is the head of
// x -> z (owner counts credit the tail x).  Order inside C(z) is immaterial.
__device__ __forceinline__ bool cand_flip(long long dx, long long dy) { return dy > dx; }

// d+ of every vertex as one int: the candidate passes read it at random, once
// per oriented edge.
__global__ void k_dplus(const long long* __restrict__ offp, int nV, int* __restrict__ dplus) {
    for (long long u = blockIdx.x * (long long)blockDim.x + threadIdx.x; u < nV;
         u += (long long)gridDim.x * blockDim.x)
        dplus[u] = (int)(offp[u + 1] - offp[u]);
}

// C(z) holds the edges that z keeps, in their order, then the flipped ones.
// Pass 1 (FILL = false): slot[p] = the place of edge p among its head's
// flipped edges, or -1 (kept, or a pad); the kept and flipped edges of each
// vertex in kept and flips; those kept of each tile's last vertex in
// last[tile].  Pass 2 writes the lists: fbase[z] is the first flipped entry
// of C(z).  A warp per merge-path tile.
// R-MAT scale 22 (64 M oriented edges): 1.9 ms both passes (a CTA per tile, an
// atomic per flipped edge in both: 3.2 ms).
template <bool FILL>
__global__ void __launch_bounds__(kB)
k_cand(const long long* __restrict__ offp, const int* __restrict__ dplus, int nV,
       const int32_t* __restrict__ fwd, int* __restrict__ kept, int* __restrict__ flips,
       int32_t* __restrict__ slot, int* __restrict__ last, const long long* __restrict__ coff,
       const long long* __restrict__ fbase, int32_t* __restrict__ cand,
       const long long* __restrict__ splits, const int32_t* __restrict__ feid,
       int32_t* __restrict__ ceid) {
    constexpr int ROWS = 4;
    const unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const long long tile = blockIdx.x * (long long)(kB / 32) + (threadIdx.x >> 5);
    const long long total = offp[nV];
    if (tile * kOrientTile >= total + nV) return;
    const WarpTile wt = warp_tile(splits, tile, kOrientTile, total, nV);
    if (wt.nitems == 0) return;
    int before = 0;   // kept edges of the tile's first vertex in earlier tiles
    if (FILL) {
        const long long p0 = offp[wt.seg0];
        if (p0 < wt.item0) {
            for (long long j = (p0 + wt.seg0) / kOrientTile + lane; j < tile; j += 32)
                before += last[j];
            before = __reduce_add_sync(kFull, before);
        }
    }
    for (long long v0 = wt.seg0; v0 <= wt.seg1; v0 += 32) {
        const long long v = v0 + lane < nV ? v0 + lane : nV;
        const long long first = offp[v];
        const long long next = v0 + 32 <= nV ? offp[v0 + 32] : total;
        const int dv = !FILL && v < nV ? dplus[v] : 0;
        const WarpWindow w = warp_window(wt, v0, first, next);
        if (w.n == 0) continue;
        const int dx = __shfl_sync(kFull, dv, w.lane_of);   // of the lane's segment
        const int id = (int)(v0 + w.lane_of);
        int send = __shfl_down_sync(kFull, w.start, 1);
        if (lane >= w.n - 1) send = w.end;
        int mine = 0;
        long long at = 0;   // the next entry of the lane's segment
        if (FILL && lane < w.n) at = coff[id] + (id == wt.seg0 ? before : 0);
        for (int r = w.begin; r < w.end; r += 32 * ROWS) {
            int y[ROWS], x[ROWS], d[ROWS], sl[ROWS];
            long long to[ROWS];
#pragma unroll
            for (int k = 0; k < ROWS; k++) {
                const int row = r + 32 * k, e = row + lane;
                y[k] = kPad;
                x[k] = d[k] = 0;
                sl[k] = -1;
                to[k] = 0;
                if (row < w.end) {   // uniform
                    const int j = warp_owner(w, row) & 31;
                    if (e < w.end) {
                        y[k] = fwd[wt.item0 + e];
                        if (FILL) sl[k] = __ldcs(slot + wt.item0 + e);
                    }
                    if (FILL) {
                        x[k] = __shfl_sync(kFull, id, j);
                        const unsigned b = __ballot_sync(kFull, y[k] != kPad && sl[k] < 0);
                        const unsigned seg = own_bits(w, send, row);
                        const unsigned sj = __shfl_sync(kFull, seg, j);
                        to[k] = __shfl_sync(kFull, at, j) + __popc(b & sj & ((1u << lane) - 1u));
                        at += __popc(b & seg);
                    } else {
                        d[k] = __shfl_sync(kFull, dx, j);
                    }
                }
            }
            if (!FILL) {
                int dy[ROWS];
#pragma unroll
                for (int k = 0; k < ROWS; k++) dy[k] = y[k] != kPad ? dplus[y[k]] : 0;
#pragma unroll
                for (int k = 0; k < ROWS; k++)
                    if (y[k] != kPad && cand_flip(d[k], dy[k])) sl[k] = atomicAdd(flips + y[k], 1);
#pragma unroll
                for (int k = 0; k < ROWS; k++) {
                    const int row = r + 32 * k, e = row + lane;
                    if (row >= w.end) break;   // uniform
                    const unsigned b = __ballot_sync(kFull, y[k] != kPad && sl[k] < 0);
                    mine += __popc(b & own_bits(w, send, row));
                    if (e < w.end) __stcs(slot + wt.item0 + e, sl[k]);
                }
            } else {
#pragma unroll
                for (int k = 0; k < ROWS; k++)
                    if (sl[k] >= 0) to[k] = fbase[y[k]] + sl[k];
#pragma unroll
                for (int k = 0; k < ROWS; k++) {
                    if (y[k] == kPad) continue;
                    cand[to[k]] = sl[k] < 0 ? y[k] : ~x[k];   // flipped: ~tail
                    if (ceid) ceid[to[k]] = feid[wt.item0 + r + 32 * k + lane];
                }
            }
        }
        if (!FILL && lane < w.n) {
            if (mine) atomicAdd(kept + id, mine);
            if (id == wt.seg1) last[tile] = mine;
        }
    }
}

// sizes of the candidate lists (n = nV + 1, the last 0), and the first flipped
// entry of each
__global__ void k_cand_sizes(const int* __restrict__ kept, const int* __restrict__ flips, int nV,
                             int* __restrict__ size) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i <= nV;
         i += (long long)gridDim.x * blockDim.x)
        size[i] = i < nV ? kept[i] + flips[i] : 0;
}

__global__ void k_cand_flip_base(const long long* __restrict__ coff, const int* __restrict__ kept,
                                 int nV, long long* __restrict__ fbase) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nV;
         i += (long long)gridDim.x * blockDim.x)
        fbase[i] = coff[i] + kept[i];
}

// ---------------------------------------------------------------------------
// Vertex-centric counting.  Every edge (u, v) of u's candidate list asks which
// w of N+(v) are in N+(u), held in shared memory in one of two forms:
//   a bitmap over the numbers that N+(u) spans (from wb on, wn bits and a zero
//   bit behind them, to which every other number is clamped): lists N+(v) of
//   kTcLong entries or more are read by the whole warp, four entries a lane
//   with one 16-byte load; the 16-byte quads of the shorter lists of 32
//   candidates are dealt to the lanes round-robin.  An entry takes about seven
//   instructions, and a quad of a short list ten more;
//   an open-addressing hash table (multiplicative hash, linear probing, load
//   factor <= 1/2, so every probe sequence ends at an empty slot) where the
//   span is too wide, or for edge supports: N+(v) is narrowed to
//   [min N+(u), max N+(u)] by two binary searches (lists sorted by number),
//   and the (v, w) pairs of 32 candidates at a time are dealt to the lanes,
//   about 40 instructions each.
// R-MAT scale 22, 11.8 G pairs, both kernels: 36.5 ms by tables alone, 24.0
// with a bitmap and pairs dealt to the lanes, 13.5 this way (k_tc_cta 8.9,
// k_tc_warp 4.6).  512 graphs (74 M oriented edges), owner counts: 13.4 ms by
// tables, 6.6 this way.  What bounds
// it: the shared-memory reads of the bits (random words: about 3.5 wavefronts a
// warp) beside 47 GB of list reads, mostly from L2.
//   k_tc_warp: one warp per vertex with d+(u) <= warp_cap (the tc.warp_cap
//              knob, at most kWarpCap, the table's capacity); vertices handed
//              out in chunks by an atomic counter; larger ones are listed;
//   k_tc_cta:  one CTA per listed vertex, table in dynamic shared memory
//              (up to kCtaCap entries), binary search of the sorted list in
//              global memory beyond that.
// ---------------------------------------------------------------------------
constexpr int kTcWarps = 8;
constexpr int kWarpCap = 512;
constexpr int kWarpTab = 2 * kWarpCap;
// Bits of a warp's bitmap, the zero one included: 8 KB a warp, three CTAs an
// SM.  512 graphs of up to 65,536 vertices: k_tc_warp 9.4 ms with 32,768 bits
// and four CTAs (half of the lists span more ids and are probed by table), 5.1
// ms this way; R-MAT scale 22: 4.7 and 4.6 ms.
constexpr unsigned kWarpBits = 65536;
// Words of shared memory per warp: the table and its filter, in whose place
// the bitmap goes, and for edge supports the edge id (u, w) of each slot.
constexpr int tc_warp_words(bool win, bool eid) {
    const int tab = kWarpTab + kWarpTab / 4 + (eid ? kWarpTab : 0);
    return win && (int)(kWarpBits / 32) > tab ? (int)(kWarpBits / 32) : tab;
}
constexpr int kCtaCap = 16384;   // largest tc.cta_table_cap: 160 KB tables
#ifndef HN_TC_PAIR_ILP
#define HN_TC_PAIR_ILP 8
#endif
constexpr int kPairIlp = HN_TC_PAIR_ILP;   // pairs in flight per lane

// Slots of a table for up to `cap` entries: the power of two >= 2*cap that a
// vertex with d+(u) = cap asks for (and no fewer than 32).
__host__ __device__ constexpr int tc_table_slots(int cap) {
    int n = 32;
    while (n < 2 * cap) n <<= 1;
    return n;
}

// Candidates of one work item of a listed vertex with d+(u) = du: about
// item_work pairs (every list it probes is at most du long), a multiple of
// 32, at least 32.
__device__ __forceinline__ int item_cands(int du, long long item_work) {
    long long c = item_work / du;
    if (c > (1 << 20)) c = 1 << 20;
    c &= ~31LL;
    return c < 32 ? 32 : (int)c;
}

__device__ __forceinline__ unsigned tc_hash(int w, int bits) {
    return ((unsigned)w * 2654435761u) >> (32 - bits);
}

// Linear probing whose home slot is the first of a 4-slot bucket (16
// bytes): a lookup reads the whole home bucket with one 128-bit load and is
// decided there unless the bucket is full and does not hold w.  Slots are
// never emptied, so a key sits before the first empty slot of its probe
// sequence.
__device__ __forceinline__ unsigned tab_home(int w, int bits) {
    return tc_hash(w, bits - 2) << 2;
}

// Inserts w; returns its slot.
__device__ __forceinline__ unsigned tab_insert(int* tab, int bits, int w) {
    unsigned mask = (1u << bits) - 1;
    unsigned h = tab_home(w, bits);
    while (true) {
        int old = atomicCAS(tab + h, -1, w);
        if (old == -1 || old == w) return h;
        h = (h + 1) & mask;
    }
}

// Filter bit of w for a table of 2^bits slots: the top bits+3 bits of the
// same product, so a filter of 8 bits per slot (2^(bits-2) words) rejects
// most absent values with one shared-memory load and no probe loop.  Its
// word index is the home bucket of w.
__device__ __forceinline__ unsigned tc_fbit(int w, int bits) {
    return ((unsigned)w * 2654435761u) >> (32 - (bits + 3));
}

__device__ __forceinline__ unsigned tab_insert_f(int* tab, unsigned* filt, int bits, int w) {
    const unsigned h = tab_insert(tab, bits, w);
    const unsigned f = tc_fbit(w, bits);
    atomicOr(filt + (f >> 5), 1u << (f & 31));
    return h;
}

// Membership of w, for lanes whose filter bit is set (`maybe`), in the home
// bucket.  `more`: the bucket is full and does not hold w, so the answer is
// tab_rest's.  `slot`: where w is, on a hit.
__device__ __forceinline__ bool tab_bucket(const int* tab, int bits, int w, bool maybe,
                                           bool& more, unsigned& slot) {
    const unsigned h = tab_home(w, bits);
    int4 q = make_int4(-1, -1, -1, -1);
    if (maybe) q = *reinterpret_cast<const int4*>(tab + h);
    const bool hit = (q.x == w) | (q.y == w) | (q.z == w) | (q.w == w);
    slot = h + (q.x == w ? 0 : q.y == w ? 1 : q.z == w ? 2 : 3);
    // slots hold vertex ids (>= 0) or -1: the bucket is full iff the OR of
    // its slots is non-negative
    more = maybe & !hit & ((q.x | q.y | q.z | q.w) >= 0);
    return hit;
}

// The probe after a full home bucket, slot by slot (the table is at most
// half full, so it meets an empty slot): w's slot, or -1.
__device__ __forceinline__ int tab_rest(const int* tab, int bits, int w) {
    const unsigned mask = (1u << bits) - 1;
    for (unsigned p = (tab_home(w, bits) + 4) & mask;; p = (p + 1) & mask) {
        const int x = tab[p];
        if (x == w) return (int)p;
        if (x == -1) return -1;
    }
}

// Owner credit: the warp's triangles found from u, added to counts[u] once
// (each triangle is found once, from its lowest vertex in the orientation).
__device__ __forceinline__ void tc_credit_owner(unsigned long long* counts, int u,
                                                unsigned long long c) {
    for (int o = 16; o; o >>= 1) c += __shfl_down_sync(0xFFFFFFFFu, c, o);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(counts + u, c);
}

struct TcView {
    const long long* offp;   // oriented offsets
    const int* dplus;        // oriented degrees (by rank the lists are padded)
    const int32_t* fwd;      // oriented lists
    const long long* coff;   // candidate-list offsets
    const int32_t* cand;     // candidate lists C(z)
    // edge-support mode (MODE 3) only:
    const int32_t* feid;     // edge id of each fwd entry
    const int32_t* ceid;     // edge id of each candidate entry
    int* esup;               // per-edge triangle counts
};

// One triangle {u, v, w} found from u: credit its three edges (MODE 3).
__device__ __forceinline__ void tc_credit_edges(int* esup, int e_uv, int e_vw, int e_uw) {
    atomicAdd(esup + e_uv, 1);
    atomicAdd(esup + e_vw, 1);
    atomicAdd(esup + e_uw, 1);
}

// One warp: every (v, w) pair of u, w in N+(v) for v in the candidate
// list C of u, probed against L = N+(u) (hash table `tab`, or binary search
// of the sorted global list L when tab == nullptr).  Candidates v are taken
// 32 at a time (in order, or groups claimed from the CTA's counter `s_next`
// when several warps share u); each lane first narrows N+(v) to
// [min N+(u), max N+(u)] by two binary searches, then the group's pairs are
// dealt round-robin to the lanes (one search over the 33-entry prefix per
// lane per group).
//
// KIND: how membership in N+(u) is decided.  kSearch: binary search of the
// sorted list; kHash: the hash table; kBits: one bit of the bitmap `win` of
// the wn numbers from wb on, which hold all of N+(u), with a zero bit behind
// them; kBitsHash: the bitmap for those numbers, the table for the others.
enum { kSearch, kHash, kBits, kBitsHash };
constexpr int kTcLong = 128;   // kBits: lists read by the whole warp from this length on
constexpr int kQuads = 4;      // kBits: 16-byte quads of short lists in flight a lane
// CTAs an SM of the bitmap-only kernel: it waits on list loads, so occupancy
// pays.  Totals (32 registers), R-MAT scale 22: 9.7 ms at 4, 9.1 at 5, 8.8 at 8;
// owner counts, which spill below 48 registers, 512 graphs: 1.43 ms at 4, 1.38 at
// 5, 1.59 at 8.  Tables in the same kernel (62 registers): 10.0 and 1.46 ms.
__host__ __device__ constexpr int bits_ctas(int mode) { return mode == 0 ? 8 : 5; }
constexpr int kWinWords = kWin / 32 + 4;   // a zero word behind the bits, 16-byte multiples

// Clears the words of a bitmap of wn bits and the zero bit behind them.
__device__ __forceinline__ void clear_bits(unsigned* win, unsigned wn, int first, int step) {
    const int quads = (int)(wn >> 7) + 1;
    for (int j = first; j < quads; j += step)
        reinterpret_cast<uint4*>(win)[j] = make_uint4(0u, 0u, 0u, 0u);
}

// Kernels' WIN: no bitmaps (lists neither aligned nor padded); bitmaps of the
// first numbers, ranked; bitmaps of the ids that N+(u) spans.
enum { kNoWin, kRankWin, kIdWin };

template <int MODE, int KIND>
__device__ __forceinline__ unsigned long long tc_vertex_warp(
    int u, const int32_t* __restrict__ L, int du, const int32_t* __restrict__ C, int dc,
    const int* tab, const unsigned* filt, const int* teid, int bits,
    int narrow_min, int* s_next, const TcView& g, int* s_pref /*33*/, long long* s_vb /*32*/,
    int* s_v /*32*/, unsigned* s_fc /*32*/, unsigned long long* __restrict__ per_vertex,
    const unsigned* win = nullptr, int wb = 0, unsigned wn = 0) {
    constexpr bool TAB = KIND == kHash || KIND == kBitsHash;
    const int lane = threadIdx.x & 31;
    const int lo_w = KIND == kBits ? 0 : L[0], hi_w = KIND == kBits ? 0 : L[du - 1];
    unsigned long long cnt = 0, cnt_u = 0;   // all hits; MODE 2: hits owned by u
    auto claim = [&](int c) {
        if (!s_next) return c + 32;
        int t = 0;
        if (lane == 0) t = atomicAdd(s_next, 1);
        return __shfl_sync(0xFFFFFFFFu, t, 0) * 32;
    };
    for (int c0 = claim(-32); c0 < dc; c0 = claim(c0)) {
        int idx = c0 + lane;
        int dx = 0, v = 0;
        bool flp = false;   // u is the head of v -> u
        long long xb = 0;
        if (idx < dc) {
            v = C[idx];
            flp = v < 0;
            if (flp) v = ~v;
            const long long b0 = g.offp[v];
            const int32_t* lst = g.fwd + b0;
            const int n = g.dplus[v];
            // [first element >= lo_w, first element > hi_w); lists of at most
            // narrow_min entries are probed whole (two dependent searches
            // cost more than the few extra filter probes)
            int lo = 0, hi = n;
            int s0 = 0;
            if (KIND != kBits && n > narrow_min) {
                while (lo < hi) { int m = (lo + hi) >> 1; if (lst[m] < lo_w) lo = m + 1; else hi = m; }
                s0 = lo;
                hi = n;
                while (lo < hi) { int m = (lo + hi) >> 1; if (lst[m] <= hi_w) lo = m + 1; else hi = m; }
            } else {
                lo = n;
            }
            xb = b0 + s0;
            dx = lo - s0;
        }
        if (KIND == kBits) {
            unsigned h = 0;
            auto test1 = [&](int w) {
                const unsigned x = min((unsigned)(w - wb), wn);
                const unsigned hit = __funnelshift_r(win[x >> 5], 0u, x) & 1u;
                h += hit;
                if (MODE == 1 && hit) atomicAdd(per_vertex + w, 1ull);
            };
            auto test = [&](const int4& q) {
                test1(q.x);
                test1(q.y);
                test1(q.z);
                test1(q.w);
            };
            const int4 none = make_int4(kPad, kPad, kPad, kPad);
            const int n4 = (dx + 3) >> 2;
            // long lists: the whole warp on one, two loads in flight
            unsigned longs = __ballot_sync(0xFFFFFFFFu, dx >= kTcLong);
            while (longs) {
                const int l = __ffs(longs) - 1;
                longs &= longs - 1;
                const int4* q = reinterpret_cast<const int4*>(g.fwd + __shfl_sync(0xFFFFFFFFu, xb, l));
                const int n = __shfl_sync(0xFFFFFFFFu, n4, l);
                h = 0;
                for (int i0 = 0; i0 < n; i0 += 64) {
                    const int i = i0 + lane;
                    const int4 a = i < n ? q[i] : none;
                    if (i0 + 32 < n) {
                        const int4 b = i + 32 < n ? q[i + 32] : none;
                        test(a);
                        test(b);
                    } else {
                        test(a);
                    }
                }
                cnt += h;
                if (MODE == 1 || MODE == 2) {
                    const unsigned all = __reduce_add_sync(0xFFFFFFFFu, h);
                    const int vl = __shfl_sync(0xFFFFFFFFu, v, l);
                    const bool fl = __shfl_sync(0xFFFFFFFFu, (int)flp, l) != 0;
                    if (lane == 0 && all) {
                        if (MODE == 1) {
                            atomicAdd(per_vertex + u, (unsigned long long)all);
                            atomicAdd(per_vertex + vl, (unsigned long long)all);
                        } else if (fl) {
                            atomicAdd(per_vertex + vl, (unsigned long long)all);
                        } else {
                            cnt_u += all;
                        }
                    }
                }
            }
            // the others: their 16-byte quads dealt to the lanes round-robin,
            // kQuads in flight a lane
            const int m4 = dx >= kTcLong ? 0 : n4;
            int incl = m4;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += y;
            }
            s_pref[lane + 1] = incl;
            if (lane == 0) s_pref[0] = 0;
            s_vb[lane] = xb;
            if (MODE == 1) s_v[lane] = v;
            if (MODE == 2) {   // the owner of v's triangles: v (flipped), or u
                s_v[lane] = idx < dc && flp ? v : -1;
                s_fc[lane] = 0;
            }
            __syncwarp();
            const int T = s_pref[32];
            if (lane < T) {
                int a = 0, b = 32;   // candidate slot of quad `lane`
                while (b - a > 1) {
                    const int mid = (a + b) >> 1;
                    if (s_pref[mid] <= lane) a = mid; else b = mid;
                }
                int end = s_pref[a + 1];
                // quad k of the group: base[k]
                const int4* base = reinterpret_cast<const int4*>(g.fwd + s_vb[a]) - s_pref[a];
                for (int k0 = lane; k0 < T; k0 += 32 * kQuads) {
                    int4 q[kQuads];
                    int va[kQuads];
#pragma unroll
                    for (int j = 0; j < kQuads; j++) {
                        const int k = k0 + 32 * j;
                        q[j] = none;
                        va[j] = a;
                        if (k < T) {
                            if (k >= end) {   // the candidate holding quad k
                                a++;
                                if (s_pref[a + 1] <= k) {
                                    int hi = 32;
                                    while (hi - a > 1) {
                                        const int mid = (a + hi) >> 1;
                                        if (s_pref[mid] <= k) a = mid; else hi = mid;
                                    }
                                }
                                end = s_pref[a + 1];
                                base = reinterpret_cast<const int4*>(g.fwd + s_vb[a]) - s_pref[a];
                            }
                            q[j] = base[k];
                            va[j] = a;
                        }
                    }
#pragma unroll
                    for (int j = 0; j < kQuads; j++) {
                        h = 0;
                        test(q[j]);
                        cnt += h;
                        if (MODE == 1 && h) {
                            atomicAdd(per_vertex + u, (unsigned long long)h);
                            atomicAdd(per_vertex + s_v[va[j]], (unsigned long long)h);
                        }
                        if (MODE == 2 && h) {
                            if (s_v[va[j]] >= 0) atomicAdd(s_fc + va[j], h);
                            else cnt_u += h;
                        }
                    }
                }
            }
            __syncwarp();
            if (MODE == 2) {   // flipped candidates own their triangles
                if (s_v[lane] >= 0 && s_fc[lane])
                    atomicAdd(per_vertex + s_v[lane], (unsigned long long)s_fc[lane]);
                __syncwarp();
            }
            continue;
        }
        int incl = dx;
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
        }
        s_pref[lane + 1] = incl;
        if (lane == 0) s_pref[0] = 0;
        s_vb[lane] = xb;
        // MODE 3 keeps the candidate's edge id (u, v) instead of v
        // MODE 3 keeps the candidate's edge id; MODE 2 the owner of its
        // triangles when that is v (flipped), else -1 (owner u)
        if (MODE == 3) s_v[lane] = idx < dc ? g.ceid[(C - g.cand) + idx] : 0;
        else if (MODE == 2) s_v[lane] = idx < dc && flp ? v : -1;
        else s_v[lane] = v;
        if (MODE == 2) s_fc[lane] = 0;
        __syncwarp();
        const int T = s_pref[32];
        if (lane < T) {
            int a = 0, b = 32;   // candidate slot of pair `lane`
            while (b - a > 1) {
                int mid = (a + b) >> 1;
                if (s_pref[mid] <= lane) a = mid; else b = mid;
            }
            int end = s_pref[a + 1];
            const int32_t* base = g.fwd + (s_vb[a] - s_pref[a]);   // pair k's w: base[k]
            // kPairIlp pairs per lane per step (k, k+32, ...): their loads
            // of w are issued together, then probed.  FULL steps (every
            // lane's kPairIlp pairs exist; uniform in the warp) skip the
            // bounds checks; the last step of a group is partial.
            unsigned c32 = 0, c32u = 0;   // hits of this group; MODE 2: those owned by u
            auto step = [&](int k0, auto full_tag) {
                constexpr bool FULL = decltype(full_tag)::value;
                int wv[kPairIlp], va[kPairIlp];
#pragma unroll
                for (int j = 0; j < kPairIlp; j++) {
                    const int k = k0 + 32 * j;
                    wv[j] = -1;
                    va[j] = a;
                    if (FULL || k < T) {
                        if (k >= end) {   // the candidate holding pair k
                            a++;
                            if (s_pref[a + 1] <= k) {
                                // short lists: k skipped several candidates;
                                // search s_pref[a..32] (s_pref[32] = T > k)
                                int hi = 32;
                                while (hi - a > 1) {
                                    int mid = (a + hi) >> 1;
                                    if (s_pref[mid] <= k) a = mid; else hi = mid;
                                }
                            }
                            end = s_pref[a + 1];
                            base = g.fwd + (s_vb[a] - s_pref[a]);
                        }
                        wv[j] = base[k];
                        va[j] = a;
                    }
                }
                // a lane's first lookup that needs probing past its home
                // bucket waits until after the step (one divergent probe
                // loop per step instead of one per pair)
                int dw = -1, da = 0, dk = 0;
                // MODE 3: the edge (v, w) of pair k of candidate slot c
                auto e_vw = [&](int c, int k) { return g.feid[s_vb[c] - s_pref[c] + k]; };
#pragma unroll
                for (int j = 0; j < kPairIlp; j++) {
                    const int w = wv[j];
                    if (!FULL && w < 0) continue;
                    bool hit;
                    int e_uw = 0;   // MODE 3: edge (u, w)
                    if (KIND == kBitsHash && (unsigned)(w - wb) < wn) {
                        const unsigned i = (unsigned)(w - wb);
                        hit = (win[i >> 5] >> (i & 31)) & 1u;
                    } else if (TAB) {
                        const unsigned f = tc_fbit(w, bits);
                        bool more;
                        unsigned slot;
                        hit = tab_bucket(tab, bits, w, (filt[f >> 5] >> (f & 31)) & 1u, more, slot);
                        if (more) {
                            if (dw < 0) {
                                dw = w;
                                da = va[j];
                                dk = k0 + 32 * j;
                            } else {
                                const int sl = tab_rest(tab, bits, w);
                                hit = sl >= 0;
                                slot = (unsigned)sl;
                            }
                        }
                        if (MODE == 3 && hit) e_uw = teid[slot];
                    } else {
                        int lo = 0, hi = du;
                        while (lo < hi) {
                            int mid = (lo + hi) >> 1;
                            if (L[mid] < w) lo = mid + 1; else hi = mid;
                        }
                        hit = lo < du && L[lo] == w;
                        if (MODE == 3 && hit) e_uw = g.feid[(L - g.fwd) + lo];
                    }
                    c32 += hit ? 1u : 0u;
                    if (MODE == 1 && hit) {
                        atomicAdd(per_vertex + w, 1ull);
                        atomicAdd(per_vertex + u, 1ull);
                        atomicAdd(per_vertex + s_v[va[j]], 1ull);
                    }
                    if (MODE == 3 && hit)
                        tc_credit_edges(g.esup, s_v[va[j]], e_vw(va[j], k0 + 32 * j), e_uw);
                    if (MODE == 2 && hit) {
                        if (s_v[va[j]] >= 0) atomicAdd(s_fc + va[j], 1u);
                        else c32u++;
                    }
                }
                if (TAB && dw >= 0) {
                    const int sl = tab_rest(tab, bits, dw);
                    if (sl >= 0) {
                        c32++;
                        if (MODE == 1) {
                            atomicAdd(per_vertex + dw, 1ull);
                            atomicAdd(per_vertex + u, 1ull);
                            atomicAdd(per_vertex + s_v[da], 1ull);
                        }
                        if (MODE == 3) tc_credit_edges(g.esup, s_v[da], e_vw(da, dk), teid[sl]);
                        if (MODE == 2) {
                            if (s_v[da] >= 0) atomicAdd(s_fc + da, 1u);
                            else c32u++;
                        }
                    }
                }
            };
            int k0 = lane;
            for (; k0 - lane + 32 * kPairIlp <= T; k0 += 32 * kPairIlp)
                step(k0, std::integral_constant<bool, true>());
            if (k0 < T) step(k0, std::integral_constant<bool, false>());
            cnt += c32;
            cnt_u += c32u;
        }
        __syncwarp();
        if (MODE == 2) {   // flipped candidates own their triangles
            if (s_v[lane] >= 0 && s_fc[lane]) atomicAdd(per_vertex + s_v[lane], (unsigned long long)s_fc[lane]);
            __syncwarp();
        }
    }
    if (MODE == 2) tc_credit_owner(per_vertex, u, cnt_u);
    return cnt;
}

// Small vertices (d+(u) <= small_du, at most small_dc candidates; used with
// the smaller-side assignment, so every probed list is at most d+(u) long):
// a thread each, merging N+(u) with each candidate's list.  No table, no
// warp-wide steps: the per-vertex overhead that dominates tiny vertices in
// the warp kernel is gone.
template <int MODE>
__global__ void __launch_bounds__(256)
k_tc_thread(TcView g, int nV, int small_du, int small_dc,
            unsigned long long* __restrict__ per_vertex,
            unsigned long long* __restrict__ total_out) {
    __shared__ unsigned long long s_sum[8];
    unsigned long long mine = 0;
    for (long long x = blockIdx.x * (long long)blockDim.x + threadIdx.x; x < nV;
         x += (long long)gridDim.x * blockDim.x) {
        const int u = (int)x;
        const long long ub = g.offp[u];
        const int du = g.dplus[u];
        const long long cb = g.coff[u];
        const int dc = (int)(g.coff[u + 1] - cb);
        if (du == 0 || dc == 0 || du > small_du || dc > small_dc) continue;
        const int32_t* A = g.fwd + ub;
        unsigned cu = 0;   // MODE 2: hits owned by u
        for (int c = 0; c < dc; c++) {
            int v = g.cand[cb + c];
            const bool flp = v < 0;
            if (flp) v = ~v;
            const long long vb = g.offp[v];
            const int dv = g.dplus[v];
            const int32_t* Bv = g.fwd + vb;
            unsigned hits = 0;
            for (int i = 0, j = 0; i < du && j < dv;) {
                const int a = A[i], b = Bv[j];
                if (a == b) {
                    hits++;
                    if (MODE == 1) {
                        atomicAdd(per_vertex + a, 1ull);
                        atomicAdd(per_vertex + u, 1ull);
                        atomicAdd(per_vertex + v, 1ull);
                    }
                    if (MODE == 3)
                        tc_credit_edges(g.esup, g.ceid[cb + c], g.feid[vb + j], g.feid[ub + i]);
                    i++;
                    j++;
                } else if (a < b) {
                    i++;
                } else {
                    j++;
                }
            }
            if (MODE == 2) {
                if (flp) { if (hits) atomicAdd(per_vertex + v, (unsigned long long)hits); }
                else cu += hits;
            }
            mine += hits;
        }
        if (MODE == 2 && cu) atomicAdd(per_vertex + u, (unsigned long long)cu);
    }
    for (int o = 16; o; o >>= 1) mine += __shfl_down_sync(0xFFFFFFFFu, mine, o);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < 8; w++) t += s_sum[w];
        if (t) atomicAdd(total_out, t);
    }
}

// With bitmaps three CTAs per SM (their 64 KB a CTA), with tables alone five
// for the plain count (48 registers, no spills), four for the modes that credit
// vertices or edges, which carry more state.
template <int MODE, int WIN>
__global__ void __launch_bounds__(kTcWarps * 32, WIN != kNoWin ? 3 : MODE == 0 ? 5 : 4)
k_tc_warp(TcView g, int nV, unsigned long long* __restrict__ per_vertex,
          unsigned long long* __restrict__ total_out,
          int* __restrict__ counters /*[0] next vertex, [1] mid, [2] huge list size*/,
          long long* __restrict__ big, long long big_cap, int warp_cap, int mid_cap,
          long long warp_work, long long item_work, int chunk, int narrow_min, int small_du,
          int small_dc) {
    extern __shared__ __align__(16) int s_dyn[];   // tc_warp_words per warp
    __shared__ int s_pref[kTcWarps][33];
    __shared__ long long s_vb[kTcWarps][32];
    __shared__ int s_v[kTcWarps][32];
    __shared__ unsigned s_fc[kTcWarps][32];   // MODE 2: hits owned by each candidate
    __shared__ unsigned long long s_sum[kTcWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int* tab = s_dyn + warp * tc_warp_words(WIN != kNoWin, MODE == 3);
    unsigned long long mine = 0;
    while (true) {
        int u0 = 0;
        if (lane == 0) u0 = atomicAdd(counters, chunk);
        u0 = __shfl_sync(0xFFFFFFFFu, u0, 0);
        if (u0 >= nV) break;
        int u1 = u0 + chunk < nV ? u0 + chunk : nV;
        for (int u = u0; u < u1; u++) {
            const long long ub = g.offp[u];
            const int du = g.dplus[u];
            const long long cb = g.coff[u];
            const int dc = (int)(g.coff[u + 1] - cb);
            if (du == 0 || dc == 0) continue;
            if (du <= small_du && dc <= small_dc) continue;   // k_tc_thread's
            // every probed list of u is at most du long: dc * du bounds u's pairs
            if (du > warp_cap || (long long)dc * du > warp_work) {
                // listed: one work item (u, chunk) per item_cands candidates;
                // mid items from the front of `big`, huge items from the back
                if (lane == 0) {
                    const int ipc = item_cands(du, item_work);
                    const int nch = (dc + ipc - 1) / ipc;
                    if (du <= mid_cap) {
                        const int p = atomicAdd(counters + 1, nch);
                        for (int c = 0; c < nch; c++) big[p + c] = ((long long)u << 32) | c;
                    } else {
                        const int p = atomicAdd(counters + 2, nch);
                        for (int c = 0; c < nch; c++)
                            big[big_cap - 1 - (p + c)] = ((long long)u << 32) | c;
                    }
                }
                continue;
            }
            // the numbers that a bitmap in the table's place would hold
            int wb = 0;
            unsigned wn = 0;
            if (WIN == kRankWin) {
                wn = (unsigned)u;
            } else if (WIN == kIdWin) {
                wb = g.fwd[ub];
                wn = (unsigned)(g.fwd[ub + du - 1] - wb) + 1u;
            }
            if (WIN != kNoWin && wn < kWarpBits) {
                unsigned* win = (unsigned*)tab;
                clear_bits(win, wn, lane, 32);
                __syncwarp();
                for (int i = lane; i < du; i += 32) {
                    const int x = g.fwd[ub + i] - wb;
                    atomicOr(win + (x >> 5), 1u << (x & 31));
                }
                __syncwarp();
                mine += tc_vertex_warp<MODE, kBits>(
                    u, g.fwd + ub, du, g.cand + cb, dc, nullptr, nullptr, nullptr, 0, narrow_min,
                    nullptr, g, s_pref[warp], s_vb[warp], s_v[warp], s_fc[warp], per_vertex, win,
                    wb, wn);
                __syncwarp();
                continue;
            }
            int bits = 32 - __clz(2 * du - 1);   // table of 2^bits >= 2*du slots
            if (bits < 5) bits = 5;
            unsigned* filt = (unsigned*)(tab + kWarpTab);
            for (int i = lane; i < (1 << bits); i += 32) tab[i] = -1;
            for (int i = lane; i < (1 << (bits - 2)); i += 32) filt[i] = 0u;
            __syncwarp();
            int* teid = MODE == 3 ? tab + kWarpTab + kWarpTab / 4 : nullptr;
            for (int i = lane; i < du; i += 32) {
                const unsigned h = tab_insert_f(tab, filt, bits, g.fwd[ub + i]);
                if (MODE == 3) teid[h] = g.feid[ub + i];
            }
            __syncwarp();
            const unsigned long long cu = tc_vertex_warp<MODE, kHash>(
                u, g.fwd + ub, du, g.cand + cb, dc, tab, filt, teid, bits, narrow_min, nullptr, g,
                s_pref[warp], s_vb[warp], s_v[warp], s_fc[warp], per_vertex);
            mine += cu;
            __syncwarp();
        }
    }
    for (int o = 16; o; o >>= 1) mine += __shfl_down_sync(0xFFFFFFFFu, mine, o);
    if (lane == 0) s_sum[warp] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < kTcWarps; w++) t += s_sum[w];
        if (t) atomicAdd(total_out, t);
    }
}

// Listed vertices (d+(u) > warp_cap): one CTA each, its warps claiming
// groups of 32 candidates from a shared counter.  Two launches (with bitmaps
// three, see WIN): the mid list
// (d+(u) <= tc.mid_cap, several CTAs per SM) and the huge list (d+(u) up to
// tc.cta_table_cap in a table, binary search of N+(u) beyond that).  A
// table of d entries takes the power of two >= 2*d slots, so the dynamic
// shared memory holds tc_table_slots(cap) slots and their filter.  The
// lists share `big` (items (u << 32) | chunk, each item_cands(d+(u))
// candidates of u): mid from the front (counters[1] entries), huge from the
// back (counters[2] entries).
// WIN: the vertices whose N+(u) fits a 16 KB bitmap (ranked, the first kWin + 1
// numbers; under ids, spans of at most kWin) are a launch of their own over both
// lists (BITS), which needs no table and fewer registers (bits_ctas an SM).  The
// others have the table, ranked with the bitmap of the members among the first
// kWin numbers in front of it.  No list exceeds `cap` (checked by the host).
template <int MODE, int WIN, bool BITS>
__global__ void __launch_bounds__(kTcWarps * 32, BITS ? bits_ctas(MODE) : 4)
k_tc_cta(TcView g, int nV, unsigned long long* __restrict__ per_vertex,
         unsigned long long* __restrict__ total_out, const int* __restrict__ counters,
         const long long* __restrict__ big, long long big_cap, long long item_work, int narrow_min,
         int huge, int cap) {
    extern __shared__ __align__(16) int s_dyn[];
    __shared__ int s_pref[kTcWarps][33];
    __shared__ long long s_vb[kTcWarps][32];
    __shared__ int s_v[kTcWarps][32];
    __shared__ unsigned s_fc[kTcWarps][32];   // MODE 2: hits owned by each candidate
    __shared__ unsigned long long s_sum[kTcWarps];
    __shared__ int s_next;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nhuge = BITS || huge ? counters[2] : 0, nmid = BITS || !huge ? counters[1] : 0;
    unsigned long long mine = 0;
    for (int i = blockIdx.x; i < nhuge + nmid; i += gridDim.x) {
        const long long item = i < nhuge ? big[big_cap - 1 - i] : big[i - nhuge];
        const int u = (int)(item >> 32);
        const int ch = (int)(item & 0xFFFFFFFF);
        const long long ub = g.offp[u];
        const int du = g.dplus[u];
        const int ipc = item_cands(du, item_work);
        const long long cb = g.coff[u] + (long long)ch * ipc;
        const int rest = (int)(g.coff[u + 1] - cb);
        const int dc = rest < ipc ? rest : ipc;
        int wb = 0;
        unsigned wn = 0;
        bool hash = du <= cap;
        if (WIN == kRankWin) {
            wn = (unsigned)min(u, kWin);
            hash = u > kWin;
        } else if (WIN == kIdWin) {
            wb = g.fwd[ub];
            wn = (unsigned)(g.fwd[ub + du - 1] - wb) + 1u;
            hash = wn > kWin;
        }
        if (WIN != kNoWin && hash == BITS) continue;   // the other launch's
        unsigned* win = (unsigned*)s_dyn;                  // BITS or ranked: kWin bits
        int* slots = s_dyn + (WIN == kRankWin ? kWinWords : 0);
        unsigned* filt = (unsigned*)(slots + tc_table_slots(cap));
        int* teid = MODE == 3 ? (int*)(filt + tc_table_slots(cap) / 4) : nullptr;
        int bits = 0;
        if (threadIdx.x == 0) s_next = 0;
        if (BITS || WIN == kRankWin) clear_bits(win, wn, threadIdx.x, blockDim.x);
        if (!BITS && hash) {
            bits = 32 - __clz(2 * du - 1);
            if (bits < 5) bits = 5;
            for (int j = threadIdx.x; j < (1 << bits); j += blockDim.x) slots[j] = -1;
            for (int j = threadIdx.x; j < (1 << (bits - 2)); j += blockDim.x) filt[j] = 0u;
        }
        if (BITS || hash) {
            __syncthreads();
            for (int j = threadIdx.x; j < du; j += blockDim.x) {
                const int w = g.fwd[ub + j];
                if (BITS || (WIN == kRankWin && w < kWin)) {
                    const int x = w - wb;
                    atomicOr(win + (x >> 5), 1u << (x & 31));
                } else {
                    const unsigned h = tab_insert_f(slots, filt, bits, w);
                    if (MODE == 3) teid[h] = g.feid[ub + j];
                }
            }
        }
        __syncthreads();
        auto run = [&](auto kind) {
            return tc_vertex_warp<MODE, decltype(kind)::value>(
                u, g.fwd + ub, du, g.cand + cb, dc, slots, filt, teid, bits, narrow_min, &s_next, g,
                s_pref[warp], s_vb[warp], s_v[warp], s_fc[warp], per_vertex, win, wb, wn);
        };
        unsigned long long cu;
        if (BITS) cu = run(std::integral_constant<int, kBits>());
        else if (WIN == kRankWin) cu = run(std::integral_constant<int, kBitsHash>());
        else if (WIN == kIdWin || hash) cu = run(std::integral_constant<int, kHash>());
        else cu = run(std::integral_constant<int, kSearch>());
        mine += cu;
        __syncthreads();
    }
    for (int o = 16; o; o >>= 1) mine += __shfl_down_sync(0xFFFFFFFFu, mine, o);
    if (lane == 0) s_sum[warp] = mine;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int w = 0; w < kTcWarps; w++) t += s_sum[w];
        if (t) atomicAdd(total_out, t);
    }
}

}  // namespace

void build_oriented(hn_graph* g, Oriented& o, const int32_t* canon) {
    cudaStream_t s = g->stream;
    const int nV = g->nV;
    const long long m = g->nE;
    o.prefix.alloc((size_t)nV + 1, s);
    degree_prefix(g, nullptr, nV, o.prefix.get());
    DevBuf<int32_t> pos((size_t)m + 1, s);
    const long long grid = (long long)g->info.sms * 8;
    DevBuf<long long> splits;
    lb_splits(g, o.prefix.get(), nV, m, Tile::TILE, splits);
    HN_LAUNCH(k_orient_flags, grid, kB, 0, s, o.prefix.get(), nV, g->vtab, g->pool, pos.get(),
              splits.get(), (long long)splits.n - 1);
    exclusive_scan(g, (const int32_t*)pos.get(), pos.get(), m + 1, s);
    // arrays of the kept edges alone, about half of m (a count above 2^31 would
    // not fit its 32 bits: the bound then)
    o.total = m;
    if (m <= INT_MAX) {
        HN_CUDA(cudaMemcpyAsync(g->h_scalar + 5, pos.get() + m, sizeof(int32_t),
                                cudaMemcpyDeviceToHost, s));
        HN_CUDA(cudaStreamSynchronize(s));
        o.total = *(const int*)(g->h_scalar + 5);
    }
    o.offp.alloc((size_t)nV + 1, s);
    o.fwd.alloc((size_t)(o.total + 4), s);
    if (canon) o.feid.alloc((size_t)(o.total + 4), s);
    HN_LAUNCH(k_orient_fill, grid, kB, 0, s, o.prefix.get(), nV, g->vtab, g->pool, pos.get(),
              o.fwd.get(), o.offp.get(), splits.get(), (long long)splits.n - 1, canon,
              canon ? o.feid.get() : (int32_t*)nullptr);
    o.dplus.alloc((size_t)nV, s);
    HN_LAUNCH(k_dplus, grid_for(g, nV, kB), kB, 0, s, (const long long*)o.offp.get(), nV,
              o.dplus.get());
}

// The orientation for bitmaps: true and o filled, or false where build_oriented
// has to do: tc.flip = 0, numbers too close to kPad, a list too long for the
// CTA kernel's table (by rank it could not be searched).  Ranked when most
// edges join vertices of more than kLocal apart in id; otherwise, as in a
// union of small graphs, ids keep the lists of neighbours close in memory,
// which ranks would scatter, and lists span few of them.
static bool build_padded(hn_graph* g, Oriented& o) {
    cudaStream_t s = g->stream;
    const int nV = g->nV;
    const long long m = g->nE;
    if (m == 0 || m > 0x7FFFFFFFll || nV > kPad - 2 * kWin || !knob(kKnobTcFlip)) return false;
    o.prefix.alloc((size_t)nV + 1, s);
    degree_prefix(g, nullptr, nV, o.prefix.get());
    int* local = (int*)(g->d_scalar + 4);   // [0] local samples, [1] longest oriented list
    HN_CUDA(cudaMemsetAsync(local, 0, 2 * sizeof(int), s));
    bool ranked = false;
    if (nV > kLocal) {
        constexpr int kSamples = 16384;
        HN_LAUNCH(k_local_sample, kSamples / 256, 256, 0, s, o.prefix.get(), nV, m, g->vtab,
                  g->pool, kSamples, local);
        HN_CUDA(cudaMemcpyAsync(g->h_scalar + 4, local, sizeof(long long), cudaMemcpyDeviceToHost, s));
        HN_CUDA(cudaStreamSynchronize(s));
        ranked = 2 * *(const int*)(g->h_scalar + 4) <= kSamples;
    }
    DevBuf<int32_t> key((size_t)nV, s);   // numbers, or degrees
    if (ranked) {   // vertices sorted by degree, stably (so by id among equals)
        o.inv.alloc((size_t)nV, s);
        DevBuf<unsigned long long> k1((size_t)nV, s), k2((size_t)nV, s);
        HN_LAUNCH(k_rank_keys, grid_for(g, nV, kB), kB, 0, s, g->vtab, nV, k1.get());
        unsigned long long *kc = k1.get(), *ka = k2.get();
        uint32_t *v1 = nullptr, *v2 = nullptr;
        HN_CUDA(cudaMemsetAsync(&g->alloc->error, 0, sizeof(int), s));
        radix_sort_u64(g, kc, ka, v1, v2, nV, 32, &g->alloc->error, s);
        check_device_error(g);   // unsorted keys are no permutation
        HN_LAUNCH(k_rank_of, grid_for(g, nV, kB), kB, 0, s, (const unsigned long long*)kc, nV,
                  key.get(), o.inv.get());
    } else {
        HN_LAUNCH(k_degree_of, grid_for(g, nV, kB), kB, 0, s, g->vtab, nV, key.get());
    }
    const long long ntiles = (m + nV + kOrientTile - 1) / kOrientTile;
    const long long grid = (ntiles + kB / 32 - 1) / (kB / 32);
    DevBuf<long long> splits;
    lb_splits(g, o.prefix.get(), nV, m, kOrientTile, splits);
    DevBuf<unsigned> kept((size_t)m / 32 + 2, s);
    DevBuf<int> last((size_t)ntiles, s);
    o.dplus.alloc((size_t)nV, s);
    DevBuf<int> cnt((size_t)nV + 1, s);
    HN_CUDA(cudaMemsetAsync(kept.get(), 0, sizeof(unsigned) * kept.n, s));
    HN_CUDA(cudaMemsetAsync(last.get(), 0, sizeof(int) * last.n, s));
    HN_CUDA(cudaMemsetAsync(o.dplus.get(), 0, sizeof(int) * (size_t)nV, s));
    auto orient = [&](auto fill) {
        auto launch = [&](auto by_rank) {
            constexpr bool FILL = decltype(fill)::value, RANKED = decltype(by_rank)::value;
            HN_LAUNCH((k_orient<FILL, RANKED>), grid, kB, 0, s, (const long long*)o.prefix.get(), nV,
                      m, (const VRec*)g->vtab, (const int32_t*)g->pool, (const int32_t*)key.get(),
                      kept.get(), o.dplus.get(), last.get(), (const long long*)o.offp.get(),
                      o.fwd.get(), (const long long*)splits.get(), ntiles);
        };
        if (ranked) launch(std::true_type());
        else launch(std::false_type());
    };
    orient(std::false_type());
    HN_LAUNCH(k_max_int, grid_for(g, nV, kB), kB, 0, s, (const int*)o.dplus.get(), nV, local + 1);
    HN_CUDA(cudaMemcpyAsync(g->h_scalar + 4, local, sizeof(long long), cudaMemcpyDeviceToHost, s));
    o.offp.alloc((size_t)nV + 1, s);
    HN_LAUNCH(k_padded, grid_for(g, (long long)nV + 1, kB), kB, 0, s, (const int*)o.dplus.get(),
              nV, cnt.get());
    exclusive_scan(g, (const int*)cnt.get(), o.offp.get(), (long long)nV + 1, s);
    HN_CUDA(cudaMemcpyAsync(g->h_scalar + 5, o.offp.get() + nV, sizeof(long long),
                            cudaMemcpyDeviceToHost, s));
    HN_CUDA(cudaStreamSynchronize(s));
    if (((const int*)(g->h_scalar + 4))[1] > knob(kKnobTcCtaTableCap)) return false;
    o.total = g->h_scalar[5];
    o.fwd.alloc((size_t)(o.total + 4), s);
    orient(std::true_type());
    HN_LAUNCH(k_pad_lists, grid_for(g, nV, kB), kB, 0, s, (const long long*)o.offp.get(),
              (const int*)o.dplus.get(), nV, o.fwd.get());
    o.prefix.release();
    o.padded = true;
    o.ranked = ranked;
    return true;
}

void build_for_counting(hn_graph* g, Oriented& o) {
    if (!build_padded(g, o)) build_oriented(g, o);
}

// C(z) for every vertex z: offsets coff (nV+1) and lists cand.
void build_candidates(hn_graph* g, const Oriented& o, DevBuf<long long>& coff,
                      DevBuf<int32_t>& cand, DevBuf<int32_t>* ceid) {
    cudaStream_t s = g->stream;
    const int nV = g->nV;
    const long long m = o.total;
    const long long ntiles = (m + nV + kOrientTile - 1) / kOrientTile;
    const long long grid = (ntiles + kB / 32 - 1) / (kB / 32);
    DevBuf<long long> splits, fbase((size_t)nV, s);
    lb_splits(g, o.offp.get(), nV, m, kOrientTile, splits);
    DevBuf<int> kept((size_t)nV, s), flips((size_t)nV, s), size((size_t)nV + 1, s);
    DevBuf<int> last((size_t)ntiles, s);
    DevBuf<int32_t> slot((size_t)m + 4, s);
    HN_CUDA(cudaMemsetAsync(kept.get(), 0, sizeof(int) * (size_t)nV, s));
    HN_CUDA(cudaMemsetAsync(flips.get(), 0, sizeof(int) * (size_t)nV, s));
    HN_CUDA(cudaMemsetAsync(last.get(), 0, sizeof(int) * last.n, s));
    coff.alloc((size_t)nV + 1, s);
    cand.alloc((size_t)m + 4, s);
    if (ceid) ceid->alloc((size_t)m + 4, s);
    auto pass = [&](auto fill) {
        constexpr bool FILL = decltype(fill)::value;
        HN_LAUNCH(k_cand<FILL>, grid, kB, 0, s, (const long long*)o.offp.get(),
                  (const int*)o.dplus.get(), nV, (const int32_t*)o.fwd.get(), kept.get(),
                  flips.get(), slot.get(), last.get(), (const long long*)coff.get(),
                  (const long long*)fbase.get(), cand.get(), (const long long*)splits.get(),
                  ceid ? (const int32_t*)o.feid.get() : (const int32_t*)nullptr,
                  ceid ? ceid->get() : (int32_t*)nullptr);
    };
    pass(std::false_type());
    HN_LAUNCH(k_cand_sizes, grid_for(g, (long long)nV + 1, kB), kB, 0, s, (const int*)kept.get(),
              (const int*)flips.get(), nV, size.get());
    exclusive_scan(g, (const int*)size.get(), coff.get(), (long long)nV + 1, s);
    HN_LAUNCH(k_cand_flip_base, grid_for(g, nV, kB), kB, 0, s, (const long long*)coff.get(),
              (const int*)kept.get(), nV, fbase.get());
    pass(std::true_type());
}

// mode 0: total only; 1: per-vertex counts (each triangle credited to its
// three vertices); 2: owner counts (each triangle credited once, to its
// lowest vertex in the degree orientation).
// Dynamic shared memory of a listed-vertex table of up to `cap` entries:
// its slots, their filter (8 bits per slot) and, for edge support, the edge
// id of each slot.
constexpr size_t tc_table_bytes(int cap, bool eid = false) {
    return (size_t)tc_table_slots(cap) * (sizeof(int) + 1 + (eid ? sizeof(int) : 0));
}
constexpr int kCtaCapEid = 8192;   // largest table with edge ids (147 KB)

template <int MODE, int WIN>
void launch_counting(hn_graph* g, const TcView& view, unsigned long long* d_counts,
                     unsigned long long* d_total, int* counters, long long* big,
                     long long big_cap, bool flipped) {
    cudaStream_t s = g->stream;
    const long long gw = (long long)g->info.sms * knob(kKnobTcWarpCtasPerSm);
    const int warp_cap = (int)knob(kKnobTcWarpCap);
    // vertices that a warp takes at a time: fewer on small graphs, where 16
    // heavy ones in a row kept one warp busy after the others had finished
    // (100,003 vertices, 2.2 M edges: 3.0 ms at 16, 0.8 at 1; 4.2 M vertices:
    // 6.6 ms at 1, 4.6 at 8 and 16)
    const int chunk = (int)std::max(1ll, std::min<long long>(knob(kKnobTcChunk),
                                                             g->nV / (g->info.sms * 512ll)));
    constexpr bool by_rank = WIN == kRankWin;
    // lists by rank are not sorted: nothing to narrow
    const int narrow_min = by_rank ? INT_MAX : (int)knob(kKnobTcNarrowMin);
    // (items of 2^20 pairs by rank instead of 2^18: R-MAT graphs of 63 and 69 M
    // edges 9.0 -> 9.3 and 8.9 -> 9.1 ms, of 128 M edges 17.2 -> 17.1)
    const long long warp_work = knob(kKnobTcWarpWork), item_work = knob(kKnobTcItemWork);
    constexpr bool eid = MODE == 3;
    const int cap_max = eid ? kCtaCapEid : kCtaCap;
    // (the bitmap holds most members: a smaller table leaves room for four CTAs
    // an SM)
    const int mid_cap = WIN != kNoWin ? (int)std::min<long long>(knob(kKnobTcMidCap), 2048)
                                : (int)knob(kKnobTcMidCap);
    const int cta_cap = (int)std::min<long long>(knob(kKnobTcCtaTableCap), cap_max);
    constexpr size_t bits = kWinWords * sizeof(int);
    constexpr size_t win = WIN == kRankWin ? bits : 0;   // in front of the tables
    const size_t dyn_mid = win + tc_table_bytes(mid_cap, eid);
    const size_t dyn_huge = win + tc_table_bytes(cta_cap, eid);
    constexpr size_t dyn_warp = sizeof(int) * kTcWarps * tc_warp_words(WIN != kNoWin, eid);
    // (set per call: the attributes belong to the device in use)
    HN_CUDA(cudaFuncSetAttribute((k_tc_cta<MODE, WIN, false>),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(win + tc_table_bytes(cap_max, eid))));
    HN_CUDA(cudaFuncSetAttribute((k_tc_warp<MODE, WIN>), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)dyn_warp));
    int mid_per_sm = 0;
    HN_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&mid_per_sm, (k_tc_cta<MODE, WIN, false>),
                                                          kTcWarps * 32, dyn_mid));
    if (mid_per_sm < 1) mid_per_sm = 1;
    // small vertices by thread (only with the smaller-side assignment, which
    // bounds every probed list by d+(u),
    // and sorted lists, which it merges)
    const int small_du = flipped && !by_rank ? (int)knob(kKnobTcThreadDu) : 0;
    const int small_dc = (int)knob(kKnobTcThreadDc);
    if (small_du > 0)
        HN_LAUNCH(k_tc_thread<MODE>, (long long)g->info.sms * 8, 256, 0, s, view, g->nV, small_du,
                  small_dc, d_counts, d_total);
    HN_LAUNCH((k_tc_warp<MODE, WIN>), gw, kTcWarps * 32, dyn_warp, s, view, g->nV, d_counts, d_total,
              counters, big, big_cap, warp_cap, mid_cap, warp_work, item_work, chunk, narrow_min,
              small_du, small_dc);
    if constexpr (WIN != kNoWin)
        HN_LAUNCH((k_tc_cta<MODE, WIN, true>), (long long)g->info.sms * bits_ctas(MODE), kTcWarps * 32, bits, s,
                  view, g->nV, d_counts, d_total, counters, big, big_cap, item_work, narrow_min, 0,
                  0);
    HN_LAUNCH((k_tc_cta<MODE, WIN, false>), (long long)g->info.sms * mid_per_sm, kTcWarps * 32,
              dyn_mid, s, view, g->nV, d_counts, d_total, counters, big, big_cap, item_work,
              narrow_min, 0, mid_cap);
    HN_LAUNCH((k_tc_cta<MODE, WIN, false>), (long long)g->info.sms, kTcWarps * 32, dyn_huge, s, view,
              g->nV, d_counts, d_total, counters, big, big_cap, item_work, narrow_min, 1, cta_cap);
}

namespace {

// mode 0: total; 1: per-vertex counts; 2: owner counts; 3: edge supports.
unsigned long long run_counting(hn_graph* g, const Oriented& o, int mode,
                                unsigned long long* d_counts, int* esup) {
    cudaStream_t s = g->stream;
    unsigned long long* d_total = (unsigned long long*)g->d_scalar;
    HN_CUDA(cudaMemsetAsync(d_total, 0, sizeof(unsigned long long), s));
    int* counters = (int*)(g->d_scalar + 1);  // next vertex, mid and huge list sizes
    HN_CUDA(cudaMemsetAsync(counters, 0, 3 * sizeof(int), s));
    // work items: at most one per vertex plus one per 32 candidates
    const long long big_cap = (long long)g->nV + g->nE / 32 + 2;
    DevBuf<long long> big((size_t)big_cap, s);
    // candidate lists: each oriented edge with the endpoint of the longer
    // out-list (owner counts credit the edge's tail, the lowest vertex of
    // the triangles it finds, which a flipped entry names)
    // (tc.flip = 0: every edge stays with its tail, C(u) = N+(u); edge
    // supports always use the lists)
    DevBuf<long long> coff;
    DevBuf<int32_t> cand, ceid;
    TcView view{o.offp.get(), o.dplus.get(), o.fwd.get(), o.offp.get(), o.fwd.get(), nullptr,
                nullptr, nullptr};
    const bool flipped = mode == 3 || knob(kKnobTcFlip);
    if (flipped) {
        build_candidates(g, o, coff, cand, mode == 3 ? &ceid : nullptr);
        view.coff = coff.get();
        view.cand = cand.get();
    }
    if (mode == 3) {
        view.feid = o.feid.get();
        view.ceid = ceid.get();
        view.esup = esup;
    }
    if (d_counts) HN_CUDA(cudaMemsetAsync(d_counts, 0, sizeof(unsigned long long) * g->nV, s));
    long long* bp = big.get();
    auto count = [&](auto m) {   // (edge supports are counted with tables)
        constexpr int M = decltype(m)::value;
        auto launch = [&](auto win) {
            launch_counting<M, decltype(win)::value>(g, view, d_counts, d_total, counters, bp,
                                                     big_cap, flipped);
        };
        if constexpr (M != 3) {
            if (o.ranked) return launch(std::integral_constant<int, kRankWin>());
            if (o.padded) return launch(std::integral_constant<int, kIdWin>());
        }
        launch(std::integral_constant<int, kNoWin>());
    };
    switch (mode) {
        case 0: count(std::integral_constant<int, 0>()); break;
        case 1: count(std::integral_constant<int, 1>()); break;
        case 2: count(std::integral_constant<int, 2>()); break;
        default: count(std::integral_constant<int, 3>());
    }
    read_scalars(g, 1);
    return (unsigned long long)g->h_scalar[0];
}

}  // namespace

unsigned long long count_triangles(hn_graph* g, const Oriented& o, unsigned long long* d_counts,
                                   int mode) {
    if (!d_counts || !o.ranked)
        return run_counting(g, o, d_counts ? mode : 0, d_counts, nullptr);
    // counted under numbers, then handed out under vertex ids
    DevBuf<unsigned long long> by_rank((size_t)g->nV, g->stream);
    const unsigned long long t = run_counting(g, o, mode, by_rank.get(), nullptr);
    HN_LAUNCH(k_unrank, grid_for(g, g->nV, kB), kB, 0, g->stream,
              (const unsigned long long*)by_rank.get(), (const int32_t*)o.inv.get(), g->nV, d_counts);
    HN_CUDA(cudaStreamSynchronize(g->stream));
    return t;
}

unsigned long long edge_support(hn_graph* g, const Oriented& o, int32_t* sup) {
    HN_REQUIRE(o.feid.get() != nullptr, "edge support needs an orientation built with edge ids");
    return run_counting(g, o, 3, nullptr, sup);
}

}  // namespace hn

using namespace hn;

extern "C" int hn_tc(hn_graph_t* g, uint64_t* per_vertex, int mem, uint64_t* total) {
    HN_API_BEGIN
    HN_REQUIRE(g != nullptr, "graph is null");
    HN_REQUIRE(mem == HN_MEM_HOST || mem == HN_MEM_DEVICE, "bad memory kind");
    HandleUse use(g);
    HN_CUDA(cudaSetDevice(g->device));
    cudaStream_t s = g->stream;
    if (g->nV == 0) {
        if (total) *total = 0;
        return HN_OK;
    }
    Oriented o;
    build_for_counting(g, o);
    DevBuf<unsigned long long> pv;
    unsigned long long* d_pv = nullptr;
    if (per_vertex) {
        if (mem == HN_MEM_HOST) {
            pv.alloc((size_t)g->nV, s);
            d_pv = pv.get();
        } else {
            d_pv = (unsigned long long*)per_vertex;
        }
    }
    unsigned long long t = count_triangles(g, o, d_pv);
    if (per_vertex && mem == HN_MEM_HOST)
        HN_CUDA(cudaMemcpyAsync(per_vertex, d_pv, sizeof(unsigned long long) * g->nV,
                                cudaMemcpyDeviceToHost, s));
    HN_CUDA(cudaStreamSynchronize(s));
    if (total) *total = t;
    HN_API_END
}

extern "C" int hn_tc_owner(hn_graph_t* g, uint64_t* counts, int mem, uint64_t* total) {
    HN_API_BEGIN
    HN_REQUIRE(g && counts, "null argument");
    HN_REQUIRE(mem == HN_MEM_HOST || mem == HN_MEM_DEVICE, "bad memory kind");
    HandleUse use(g);
    HN_CUDA(cudaSetDevice(g->device));
    cudaStream_t s = g->stream;
    if (g->nV == 0) {
        if (total) *total = 0;
        return HN_OK;
    }
    Oriented o;
    build_for_counting(g, o);
    DevBuf<unsigned long long> buf;
    unsigned long long* d_c = (unsigned long long*)counts;
    if (mem == HN_MEM_HOST) {
        buf.alloc((size_t)g->nV, s);
        d_c = buf.get();
    }
    unsigned long long t = count_triangles(g, o, d_c, 2);
    if (mem == HN_MEM_HOST)
        HN_CUDA(cudaMemcpyAsync(counts, d_c, sizeof(unsigned long long) * g->nV,
                                cudaMemcpyDeviceToHost, s));
    HN_CUDA(cudaStreamSynchronize(s));
    if (total) *total = t;
    HN_API_END
}
