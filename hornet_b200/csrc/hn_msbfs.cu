// Batched BFS: up to 64 BFS "slots" in one traversal (bit-parallel
// multi-source BFS after Then et al., "The More the Merrier: Efficient
// Multi-Source Graph Traversal", VLDB 2015).
//
// Batching: many BFS sources (and, on a disjoint union, many small graphs)
// in one launch of a CUDA graph (two where pulls are asked for).  Each vertex carries three 64-bit masks:
//   seen[v]  slots that have reached v,
//   front[v] slots for which v is on the current frontier,
//   nxt[v]   slots that reach v at this level (OR-accumulated).
// One level is two kernels inside the graph's WHILE body:
//   push:  the frontier's edges (u, v), load-balanced in chunks exactly as
//          the single-source top-down kernel does, OR front[u] & ~seen[v]
//          into nxt[v]; the first writer of nxt[v] records v as touched;
//   apply: every touched v takes its new bits, writes dist[slot][v] = level
//          for each, and joins the next frontier once (whatever the number
//          of slots) with its edge offset from one packed atomic per CTA.
// An edge is read once per level for ALL slots on it, so a 64-source batch
// reads each vertex's adjacency about as many times as there are distinct
// distances to it, instead of 64 times.  Distances per slot equal a
// single-source BFS from that slot's source; slots shared by several sources
// give the distance to the nearest of them, which is each source's own
// distance when they sit in different components (a disjoint union of
// graphs, one source per graph per slot).
#include "hn_graph.cuh"
#include "hn_window.cuh"

namespace hn {

constexpr int kSeedBlock = 256;       // the single seeding CTA
constexpr int kMsChunk = 2048;        // edges per chunk (block x items per thread)
constexpr int kMaxSlots = 64;

// A level pushes and applies the touched vertices it listed, pulls (apply
// does the work), or pushes without a list and applies in a pass over all
// vertices.  A pull looks for a vertex's predecessors in its own list, so it
// is right only where every edge is stored both ways: the first level that
// would pull leaves the loop, the host has the edges checked (k_ms_one_way)
// and goes on with the loop, pulling or not.
enum { kMsPush, kMsPull, kMsPushAll };

struct MsState {
    unsigned long long cnt[3];      // frontier counters: (edge total << 32) | size
    unsigned long long tcnt;        // touched vertices this level
    int level;
    unsigned ticket;
    int nV;
    int nslots;
    const VRec* vtab;
    const int32_t* pool;
    int32_t* q[2];
    long long* qbase[2];
    unsigned* qoff[2];
    int32_t* chunk[2];
    ulonglong2* sn;                 // {seen, nxt} of each vertex, one load for both
    unsigned long long* front[2];
    int32_t* touched;
    int32_t* dist;                  // nslots x nV, slot-major
    const int32_t* src;
    const int32_t* slot;
    int nsrc;
    int mode;                       // kMsPush, kMsPull or kMsPushAll
    unsigned long long* stat;       // [3*kMaxSlots]: visited, scanned, last level per slot
    int prev_nq;                    // size of the previous frontier (its fronts are cleared)
    int bottom_up;                  // bottom-up levels allowed
    int alpha, beta;                // direction switch thresholds
    long long nE;                   // edges of the graph
    long long check_min;            // edges of a frontier that the check is made for
    long long open_edges;           // degrees of the vertices that miss a slot
    unsigned long long all_mask;    // slots that hold at least one source
    int symmetric;                  // 1: every edge is stored both ways, 0: not known, -1: no
    int ask;                        // the loop has ended to have that found out
    unsigned long long one_way;     // sum over the edges, 0 when symmetric
};

struct MsGraph {
    int nV = -1;
    long long nchunk_cap = 0;
    MsState* state = nullptr;
    MsState* h_state = nullptr;
    int32_t* qbuf = nullptr;
    long long* qbasebuf = nullptr;
    unsigned* qoffbuf = nullptr;
    int32_t* chunkbuf = nullptr;
    unsigned long long* masks = nullptr;   // {seen, nxt} pairs, front0, front1
    int32_t* touched = nullptr;
    unsigned long long* stat = nullptr;
    unsigned long long* h_stat = nullptr;
    cudaGraph_t graph[2] = {nullptr, nullptr};      // [0] from the start, [1] the next levels
    cudaGraphExec_t exec[2] = {nullptr, nullptr};
    int block = 256;      // msbfs.block knob baked into the graph
    unsigned grid = 0;    // msbfs.ctas_per_sm x SMs
};

namespace {

__device__ __forceinline__ void ms_mark_chunks(int32_t* chunk, unsigned off, unsigned d, int pos) {
    unsigned c0 = (off + kMsChunk - 1) / kMsChunk;
    unsigned c1 = (off + d - 1) / kMsChunk;
    for (unsigned c = c0; c <= c1; c++) chunk[c] = pos;
}

// CTA-wide exclusive scan of a packed (degree << 32 | count) value and one
// atomic on `counter`; returns this thread's (slot, edge offset) base.
// Must be called by all threads of a BLOCK-thread CTA.
template <int BLOCK>
__device__ __forceinline__ unsigned long long ms_cta_reserve(unsigned long long mine,
                                                             unsigned long long* counter,
                                                             unsigned long long* s_wsum,
                                                             unsigned long long* s_base) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += x;
    }
    if (lane == 31) s_wsum[warp] = incl;
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned long long v = threadIdx.x < BLOCK / 32 ? s_wsum[threadIdx.x] : 0ull;
        unsigned long long vi = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long x = __shfl_up_sync(0xFFFFFFFFu, vi, o);
            if (lane >= o) vi += x;
        }
        if (threadIdx.x < BLOCK / 32) s_wsum[threadIdx.x] = vi - v;
        unsigned long long tot = __shfl_sync(0xFFFFFFFFu, vi, 31);
        if (threadIdx.x == 0) *s_base = tot ? atomicAdd(counter, tot) : 0ull;
    }
    __syncthreads();
    unsigned long long r = *s_base + s_wsum[warp] + (incl - mine);
    __syncthreads();   // s_wsum / s_base are reused by the next call
    return r;
}

__global__ void k_ms_fill(MsState* st) {
    const long long n = st->nV;
    const long long nd = n * st->nslots;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nd;
         i += (long long)gridDim.x * blockDim.x) {
        st->dist[i] = kInf;
        if (i < n) {
            st->sn[i] = make_ulonglong2(0ull, 0ull);
            st->front[0][i] = 0;
            st->front[1][i] = 0;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x < 3 * kMaxSlots) st->stat[threadIdx.x] = 0;
}

// one CTA: seed every source, build the first frontier
__global__ void __launch_bounds__(kSeedBlock) k_ms_seed(MsState* st) {
    __shared__ unsigned long long s_wsum[kSeedBlock / 32];
    __shared__ unsigned long long s_base;
    __shared__ unsigned long long s_stat[2 * kMaxSlots];
    for (int i = threadIdx.x; i < 2 * kMaxSlots; i += kSeedBlock) s_stat[i] = 0;
    if (threadIdx.x == 0) {
        st->cnt[0] = 0;
        st->cnt[1] = 0;
        st->cnt[2] = 0;
        st->tcnt = 0;
        st->level = 1;
        st->ticket = 0;
    }
    __syncthreads();
    const int nV = st->nV;
    for (int j0 = 0; j0 < st->nsrc; j0 += kSeedBlock) {
        int j = j0 + threadIdx.x;
        bool first = false;
        int v = 0;
        VRec r;
        r.deg = 0;
        r.off = 0;
        if (j < st->nsrc) {
            v = st->src[j];
            int b = st->slot ? st->slot[j] : j;
            unsigned long long bit = 1ull << b;
            atomicOr(&st->all_mask, bit);
            unsigned long long old = atomicOr(st->front[0] + v, bit);
            unsigned long long olds = atomicOr(&st->sn[v].x, bit);
            first = old == 0;
            r = st->vtab[v];
            if (!(olds & bit)) {
                st->dist[(long long)b * nV + v] = 0;
                atomicAdd(&s_stat[b], 1ull);
                atomicAdd(&s_stat[kMaxSlots + b], (unsigned long long)r.deg);
            }
        }
        bool q = first && r.deg > 0;
        unsigned long long mine = q ? (((unsigned long long)r.deg << 32) | 1ull) : 0ull;
        unsigned long long at = ms_cta_reserve<kSeedBlock>(mine, &st->cnt[0], s_wsum, &s_base);
        if (q) {
            int pos = (int)(at & 0xFFFFFFFFull);
            unsigned off = (unsigned)(at >> 32);
            st->q[0][pos] = v;
            st->qbase[0][pos] = r.off;
            st->qoff[0][pos] = off;
            ms_mark_chunks(st->chunk[0], off, (unsigned)r.deg, pos);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long c = st->cnt[0];
        st->qoff[0][c & 0xFFFFFFFFull] = (unsigned)(c >> 32);
    }
    for (int i = threadIdx.x; i < 2 * kMaxSlots; i += kSeedBlock)
        if (s_stat[i]) atomicAdd(st->stat + i, s_stat[i]);
}

// push: OR frontier masks along the frontier's edges
template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK) k_ms_push(MsState* st) {
    constexpr int IPT = kMsChunk / BLOCK;
    __shared__ unsigned s_start[kMsChunk + 2];
    __shared__ long long s_base[kMsChunk + 1];
    __shared__ unsigned long long s_front[kMsChunk + 1];
    __shared__ int s_nw;
    __shared__ unsigned long long s_wsum[BLOCK / 32];
    __shared__ unsigned long long s_cb;
    const int it = st->level - 1;
    const unsigned long long cin = st->cnt[it % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) st->cnt[(it + 2) % 3] = 0;
    const int nq = (int)(cin & 0xFFFFFFFFull);
    const unsigned total = (unsigned)(cin >> 32);
    const int cur = it & 1;
    {
        // the previous frontier's masks are spent: its buffer is the one this
        // level's apply writes, and bottom-up levels read every vertex's mask
        const int pn = st->prev_nq;
        const int32_t* pq = st->q[cur ^ 1];
        unsigned long long* pf = st->front[cur ^ 1];
        for (long long i = blockIdx.x * (long long)BLOCK + threadIdx.x; i < pn;
             i += (long long)gridDim.x * BLOCK)
            pf[pq[i]] = 0ull;
    }
    if (st->mode == kMsPull) return;   // apply does the work
    const bool listed = st->mode == kMsPush;
    const int32_t* q = st->q[cur];
    const long long* qbase = st->qbase[cur];
    const unsigned* qoff = st->qoff[cur];
    const int32_t* chunk = st->chunk[cur];
    const unsigned long long* front = st->front[cur];
    ulonglong2* sn = st->sn;
    const int32_t* pool = st->pool;
    const unsigned nchunks = (total + kMsChunk - 1) / kMsChunk;
    for (unsigned c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const unsigned e0 = c * kMsChunk;
        const unsigned e1 = e0 + kMsChunk < total ? e0 + kMsChunk : total;
        const int s0 = chunk[c];
        const int s1 = c + 1 < nchunks ? chunk[c + 1] : nq - 1;
        const int nw = s1 - s0 + 1;
        for (int j = threadIdx.x; j <= nw; j += BLOCK) {
            int s = s0 + j;
            unsigned so = qoff[s];
            s_start[j] = so;
            if (j < nw) {
                s_base[j] = qbase[s] - (long long)so;
                s_front[j] = front[q[s]];
            }
        }
        if (threadIdx.x == 0) s_nw = nw;
        __syncthreads();
        const unsigned a = e0 + threadIdx.x * IPT;
        const unsigned b = a + IPT < e1 ? a + IPT : e1;
        int touched_here[IPT];
        int nt = 0;
        if (a < b) {
            int lo = 0, hi = s_nw;
            while (hi - lo > 1) {
                int mid = (lo + hi) >> 1;
                if (s_start[mid] <= a) lo = mid; else hi = mid;
            }
            int j = lo;
            int w[IPT];
            unsigned long long fm[IPT];
#pragma unroll
            for (int k = 0; k < IPT; k++) {
                unsigned e = a + k;
                w[k] = -1;
                fm[k] = 0;
                if (e < b) {
                    while (s_start[j + 1] <= e) j++;
                    w[k] = __ldg(pool + s_base[j] + e);
                    fm[k] = s_front[j];
                }
            }
            // bits that an earlier edge of this level has already set in nxt
            // need no atomic (through L2: an L1 copy would miss them)
            unsigned long long sv[IPT];
#pragma unroll
            for (int k = 0; k < IPT; k++) {
                sv[k] = ~0ull;
                if (w[k] >= 0) {
                    const ulonglong2 q = __ldcg(sn + w[k]);
                    sv[k] = q.x | q.y;
                }
            }
#pragma unroll
            for (int k = 0; k < IPT; k++) {
                unsigned long long m = fm[k] & ~sv[k];
                if (m) {
                    if (listed) {
                        unsigned long long old = atomicOr(&sn[w[k]].y, m);
                        if (old == 0) touched_here[nt++] = w[k];
                    } else {
                        atomicOr(&sn[w[k]].y, m);
                    }
                }
            }
        }
        // nothing newly touched in the whole chunk (common late in the
        // traversal): skip the scan; the barrier still guards the window
        if (__syncthreads_or(nt > 0)) {
            unsigned long long at =
                ms_cta_reserve<BLOCK>((unsigned long long)nt, &st->tcnt, s_wsum, &s_cb);
            int pos = (int)at;
            for (int k = 0; k < nt; k++) st->touched[pos + k] = touched_here[k];
        }
    }
}

// Bottom-up step of one warp: lane's vertex (record r, missing slots `todo`)
// takes, for every slot it still misses, the frontier mask of a neighbour on
// that slot's frontier.  The first kMsLane neighbours are read by the lane
// itself, four at a time (neighbour ids with one 16-byte load, then their
// masks together); a list that needs more is read by the whole warp, 64
// neighbours a step, so a hub costs its warp deg / 64 steps instead of deg.
// Stops at the step after which nothing is missing.  Called by all lanes.
constexpr int kMsLane = 16;
constexpr long long kMsScan = 4;
// Edges of a frontier that may touch more than one in kMsAll vertices are
// pushed without a list of the touched: a pass over all vertices reads their
// masks in order, writes distances to neighbouring words and queues the next
// frontier in vertex order, where the list's order is that of the edges.
constexpr long long kMsAll = 4;

__device__ __forceinline__ unsigned long long ms_pull(const VRec& r, unsigned long long todo,
                                                      const int32_t* __restrict__ pool,
                                                      const unsigned long long* __restrict__ front) {
    const unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    unsigned long long got = 0;
    const int32_t* nb = pool + r.off;
    if (todo) {
        // blocks of capacity >= 4 are 16-byte aligned and whole
        const int mine = r.deg < kMsLane ? r.deg : kMsLane;
        for (int e = 0; e < mine; e += 4) {
            int4 n4;
            if (r.cap >= 4) n4 = __ldg(reinterpret_cast<const int4*>(nb + e));
            else n4 = make_int4(__ldg(nb), r.deg > 1 ? __ldg(nb + 1) : 0, 0, 0);   // cap 1 or 2
            const int left = r.deg - e;
            const unsigned long long m0 = front[n4.x];
            const unsigned long long m1 = left > 1 ? front[n4.y] : 0ull;
            const unsigned long long m2 = left > 2 ? front[n4.z] : 0ull;
            const unsigned long long m3 = left > 3 ? front[n4.w] : 0ull;
            got |= m0 | m1 | m2 | m3;
            if (!(todo & ~got)) break;
        }
    }
    got &= todo;
    unsigned more = __ballot_sync(kFull, r.deg > kMsLane && (todo & ~got) != 0);
    while (more) {
        const int l = __ffs(more) - 1;
        more &= more - 1;
        const int32_t* wn = pool + __shfl_sync(kFull, r.off, l);
        const int wd = __shfl_sync(kFull, r.deg, l);
        const unsigned long long wt = __shfl_sync(kFull, todo & ~got, l);
        unsigned long long acc = 0;
        for (int e = kMsLane; e < wd; e += 64) {
            const int e0 = e + lane, e1 = e + 32 + lane;
            const int a = e0 < wd ? __ldg(wn + e0) : -1;
            const int b = e1 < wd ? __ldg(wn + e1) : -1;
            const unsigned long long m = (a >= 0 ? front[a] : 0ull) | (b >= 0 ? front[b] : 0ull);
            const unsigned lo = __reduce_or_sync(kFull, (unsigned)(m & wt));
            const unsigned hi = __reduce_or_sync(kFull, (unsigned)((m & wt) >> 32));
            acc |= ((unsigned long long)hi << 32) | lo;
            if (!(wt & ~acc)) break;
        }
        if (lane == l) got |= acc;
    }
    return got;
}

// apply: new bits of every touched vertex (listed, or all vertices with bits
// in nxt) or of every vertex that misses a slot (pull), their distances, the
// next frontier.  kMsApply
// vertices per thread share one CTA-wide reservation.  Per-slot statistics
// stay in registers (lane b counts slots b and b + 32, by ballot and warp
// sum): an atomic per (vertex, slot), 64-bit and on few shared words, had
// taken most of a level.  512 graphs (8.0 M vertices, 148 M edges), 8 slots:
// 54.8 ms before, 22.3 ms with these two (lists by warps, statistics in
// registers), 7.1 ms with {seen, nxt} in one load ahead of each atomic and
// the direction chosen by the edges that either would read, 4.5 ms with the
// large levels applied in vertex order.
constexpr int kMsApply = 4;

template <int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1024 / BLOCK)
k_ms_apply(MsState* st, cudaGraphConditionalHandle cond) {
    const unsigned kFull = 0xFFFFFFFFu;
    __shared__ unsigned long long s_wsum[BLOCK / 32];
    __shared__ unsigned long long s_cb;
    __shared__ unsigned long long s_stat[2 * kMaxSlots];
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < 2 * kMaxSlots; i += BLOCK) s_stat[i] = 0;
    __syncthreads();
    const int level = st->level;
    const int it = level - 1;
    const int nx = (it & 1) ^ 1;
    unsigned long long* cout = &st->cnt[(it + 1) % 3];
    const long long nt = (long long)st->tcnt;
    const int nV = st->nV;
    const VRec* __restrict__ vtab = st->vtab;
    const int32_t* __restrict__ pool = st->pool;
    ulonglong2* sn = st->sn;
    unsigned long long* nfront = st->front[nx];
    const int mode = st->mode;
    const bool bu = mode == kMsPull;
    const unsigned long long* cfront = st->front[nx ^ 1];
    const unsigned long long all = st->all_mask;
    const int nq_in = (int)(st->cnt[it % 3] & 0xFFFFFFFFull);
    const long long n_items = mode == kMsPush ? nt : (long long)nV;
    int32_t* dist = st->dist;
    unsigned long long vis0 = 0, vis1 = 0, sc0 = 0, sc1 = 0;   // slots lane, lane + 32
    long long closed = 0;   // degrees of vertices that miss no slot any more
    constexpr long long PER = (long long)BLOCK * kMsApply;
    for (long long i0 = blockIdx.x * PER; i0 < n_items; i0 += (long long)gridDim.x * PER) {
        int vk[kMsApply], dk[kMsApply];
        long long ok[kMsApply];
        unsigned long long mine = 0;   // (degree sum << 32) | queued vertices
#pragma unroll
        for (int k = 0; k < kMsApply; k++) {
            const long long i = i0 + k * BLOCK + threadIdx.x;
            int v = 0;
            VRec r;
            r.deg = 0;
            r.off = 0;
            r.cap = 0;
            unsigned long long nw = 0;
            if (bu) {
                unsigned long long sv = 0, todo = 0;
                if (i < n_items) {
                    v = (int)i;
                    sv = sn[v].x;
                    todo = all & ~sv;
                    if (todo) {
                        r = vtab[v];
                        if (r.deg == 0) todo = 0;
                    }
                }
                nw = ms_pull(r, todo, pool, cfront);
                if (nw) {
                    sn[v].x = sv | nw;
                    nfront[v] = nw;
                    if (!(all & ~(sv | nw))) closed += r.deg;
                }
            } else if (i < n_items) {
                v = mode == kMsPush ? st->touched[i] : (int)i;
                const ulonglong2 q = sn[v];
                if (q.y) {   // (always, of a touched vertex)
                    nw = q.y & ~q.x;
                    sn[v] = make_ulonglong2(q.x | nw, 0ull);
                    nfront[v] = nw;
                    r = vtab[v];
                    if (!(all & ~(q.x | nw))) closed += r.deg;
                }
            }
            // the slots that reach any of the warp's vertices now
            unsigned ulo = __reduce_or_sync(kFull, (unsigned)nw);
            unsigned uhi = __reduce_or_sync(kFull, (unsigned)(nw >> 32));
            while (ulo | uhi) {
                const bool low = ulo != 0;
                const int b5 = __ffs(low ? ulo : uhi) - 1;
                if (low) ulo &= ulo - 1; else uhi &= uhi - 1;
                const int bb = low ? b5 : b5 + 32;
                const bool has = (nw >> bb) & 1ull;
                if (has) dist[(long long)bb * nV + v] = level;
                const unsigned c = __popc(__ballot_sync(kFull, has));
                // distinct vertices: their degrees sum to at most nE < 2^32
                const unsigned ds = __reduce_add_sync(kFull, has ? (unsigned)r.deg : 0u);
                if (lane == b5) {
                    if (low) { vis0 += c; sc0 += ds; }
                    else { vis1 += c; sc1 += ds; }
                }
            }
            const bool q = nw != 0 && r.deg > 0;
            vk[k] = v;
            dk[k] = q ? r.deg : 0;
            ok[k] = r.off;
            if (q) mine += ((unsigned long long)r.deg << 32) | 1ull;
        }
        if (!__syncthreads_or(mine != 0)) continue;   // nothing queued by the CTA
        unsigned long long at = ms_cta_reserve<BLOCK>(mine, cout, s_wsum, &s_cb);
#pragma unroll
        for (int k = 0; k < kMsApply; k++) {
            if (dk[k]) {
                const int pos = (int)(at & 0xFFFFFFFFull);
                const unsigned off = (unsigned)(at >> 32);
                st->q[nx][pos] = vk[k];
                st->qbase[nx][pos] = ok[k];
                st->qoff[nx][pos] = off;
                ms_mark_chunks(st->chunk[nx], off, (unsigned)dk[k], pos);
                at += ((unsigned long long)dk[k] << 32) | 1ull;
            }
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) closed += __shfl_xor_sync(kFull, closed, o);
    if (lane == 0 && closed)
        atomicAdd((unsigned long long*)&st->open_edges, (unsigned long long)-closed);
    if (vis0) { atomicAdd(&s_stat[lane], vis0); atomicAdd(&s_stat[kMaxSlots + lane], sc0); }
    if (vis1) { atomicAdd(&s_stat[lane + 32], vis1); atomicAdd(&s_stat[kMaxSlots + lane + 32], sc1); }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * kMaxSlots; i += BLOCK)
        if (s_stat[i]) {
            atomicAdd(st->stat + i, s_stat[i]);
            if (i < kMaxSlots) st->stat[2 * kMaxSlots + i] = (unsigned long long)level;
        }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned tk = atomicAdd(&st->ticket, 1u);
        if (tk == gridDim.x - 1) {
            __threadfence();
            unsigned long long c = atomicAdd(cout, 0ull);
            unsigned nn = (unsigned)(c & 0xFFFFFFFFull);
            st->qoff[nx][nn] = (unsigned)(c >> 32);
            st->ticket = 0;
            st->tcnt = 0;
            st->level = level + 1;
            st->prev_nq = nq_in;
            // pull while the next frontier's edges (which a push reads) exceed
            // those of the vertices that still miss a slot (which a pull reads
            // at most) -- alpha / kMsScan, about 1 by default -- and the
            // frontier holds nV/beta vertices or more.  The check for symmetry
            // reads all edges and takes a round trip to the host (60 us on a
            // small graph, 0.58 ms at 128 M edges), so a frontier of fewer than
            // check_min edges or a quarter of the graph's is pushed instead
            // (16 M edges: 8 slots 490 us pushed, 433 checked and pulled, one
            // slot 335 and 368; 8 M edges, 8 slots: 331 and 362; 128 M edges, 8
            // slots: 2.40 and 1.73 ms)
            const long long mf = (long long)(c >> 32);
            const bool more = nn > 0 && level < nV;
            int next = mf * kMsAll > nV ? kMsPushAll : kMsPush;
            int ask = 0;
            if (st->bottom_up && st->symmetric >= 0 && more) {
                const long long open = (long long)atomicAdd((unsigned long long*)&st->open_edges, 0ull);
                if (mf * st->alpha > kMsScan * open && (long long)nn * st->beta >= nV) {
                    if (st->symmetric) next = kMsPull;
                    else if (mf >= st->check_min && 4 * mf >= st->nE) ask = 1;
                }
            }
            st->mode = next;
            st->ask = ask;
            cudaGraphSetConditional(cond, more && !ask ? 1u : 0u);
        }
    }
}

// Is every edge stored both ways?  The sum over the edges (u, v) of
// mix64({min, max}), counted negative where u > v: 0 when each pair is stored
// as often one way as the other.  A single one-way edge never gives 0, others
// with a probability of 2^-64.  Loops do not count.  A warp per merge-path
// tile, windows of 32 vertices, four rows of 32 edges in flight; bound by HBM
// (4 bytes an edge).
constexpr int kMsTile = 1024;
constexpr int kOneWayBlock = 256;

__global__ void __launch_bounds__(kOneWayBlock)
k_ms_one_way(const long long* __restrict__ prefix, int nV, long long nE,
             const VRec* __restrict__ vtab, const int32_t* __restrict__ pool,
             const long long* __restrict__ splits, long long ntiles, MsState* st) {
    constexpr int ROWS = 4;
    const unsigned kFull = 0xFFFFFFFFu;
    __shared__ unsigned long long s_sum[kOneWayBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long nwarps = (long long)gridDim.x * (kOneWayBlock / 32);
    unsigned long long sum = 0;
    for (long long tile = blockIdx.x * (long long)(kOneWayBlock / 32) + warp; tile < ntiles;
         tile += nwarps) {
        const WarpTile wt = warp_tile(splits, tile, kMsTile, nE, nV);
        if (wt.nitems == 0) continue;
        for (long long v0 = wt.seg0; v0 <= wt.seg1; v0 += 32) {
            const long long v = v0 + lane < nV ? v0 + lane : nV;
            const long long first = prefix[v];
            const long long next = v0 + 32 <= nV ? prefix[v0 + 32] : nE;
            const long long off = v < nV ? vtab[v].off : 0;
            const WarpWindow w = warp_window(wt, v0, first, next);
            if (w.n == 0) continue;
            const long long base = __shfl_sync(kFull, off - first, w.lane_of) + wt.item0;
            const int id = (int)v0 + w.lane_of;
            for (int r = w.begin; r < w.end; r += 32 * ROWS) {
                int x[ROWS], u[ROWS];
#pragma unroll
                for (int k = 0; k < ROWS; k++) {
                    const int row = r + 32 * k;
                    x[k] = u[k] = 0;
                    if (row >= w.end) continue;   // uniform
                    const int j = warp_owner(w, row) & 31;
                    const long long b = __shfl_sync(kFull, base, j);
                    u[k] = __shfl_sync(kFull, id, j);
                    x[k] = row + lane < w.end ? __ldcs(pool + b + row + lane) : u[k];
                }
#pragma unroll
                for (int k = 0; k < ROWS; k++) {
                    const unsigned lo = (unsigned)min(x[k], u[k]), hi = (unsigned)max(x[k], u[k]);
                    const unsigned long long h = mix64((unsigned long long)lo << 32 | hi);
                    if (u[k] < x[k]) sum += h;
                    if (u[k] > x[k]) sum -= h;
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
    if (lane == 0) s_sum[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < kOneWayBlock / 32; i++) sum += s_sum[i];
        if (sum) atomicAdd(&st->one_way, sum);
    }
}

// One thread: the answer, and with it the direction of the level asked for.
__global__ void k_ms_answer(MsState* st) {
    st->symmetric = st->one_way ? -1 : 1;
    if (!st->one_way) st->mode = kMsPull;
    st->ask = 0;
}

void check_symmetry(hn_graph* g, MsGraph& mg) {
    cudaStream_t s = g->stream;
    try {
        DevBuf<long long> prefix((size_t)g->nV + 1, s), splits;
        degree_prefix(g, nullptr, g->nV, prefix.get());
        lb_splits(g, prefix.get(), g->nV, g->nE, kMsTile, splits);
        const long long ntiles = (g->nE + g->nV + kMsTile - 1) / kMsTile;
        HN_LAUNCH(k_ms_one_way, grid_for(g, ntiles, kOneWayBlock / 32), kOneWayBlock, 0, s,
                  (const long long*)prefix.get(), g->nV, (long long)g->nE, (const VRec*)g->vtab,
                  (const int32_t*)g->pool, (const long long*)splits.get(), ntiles, mg.state);
    } catch (const Error& e) {
        if (e.code != HN_ERR_OOM) throw;
        // no room for the check (8 bytes a vertex): as if there were one-way edges
        HN_CUDA(cudaMemsetAsync(&mg.state->one_way, 1, sizeof(mg.state->one_way), s));
    }
    HN_LAUNCH(k_ms_answer, 1, 1, 0, s, mg.state);
}

// The CUDA graph of part 0 (fill, seed and the levels) or 1 (the levels from
// where they stand, built when a call first asks).
void build_ms_loop(hn_graph* g, MsGraph& mg, int part) {
    cudaGraph_t& graph = mg.graph[part];
    if (graph) HN_CUDA(cudaGraphDestroy(graph));   // (of a build that failed)
    graph = nullptr;
    HN_CUDA(cudaGraphCreate(&graph, 0));
    cudaGraphNode_t fill, seed, condn, push, apply;
    void* args[] = {&mg.state};
    cudaKernelNodeParams p = {};
    p.kernelParams = args;
    if (part == 0) {
        p.func = (void*)k_ms_fill;
        p.gridDim = dim3((unsigned)g->info.sms * 8);
        p.blockDim = dim3(256);
        HN_CUDA(cudaGraphAddKernelNode(&fill, graph, nullptr, 0, &p));
        p.func = (void*)k_ms_seed;
        p.gridDim = dim3(1);
        p.blockDim = dim3(kSeedBlock);
        HN_CUDA(cudaGraphAddKernelNode(&seed, graph, &fill, 1, &p));
    }
    cudaGraphConditionalHandle handle;
    HN_CUDA(cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = handle;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    HN_CUDA(cudaGraphAddNode(&condn, graph, part == 0 ? &seed : nullptr, part == 0 ? 1 : 0, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    p.func = mg.block == 128 ? (void*)k_ms_push<128>
           : mg.block == 512 ? (void*)k_ms_push<512> : (void*)k_ms_push<256>;
    p.gridDim = dim3(mg.grid);
    p.blockDim = dim3(mg.block);
    HN_CUDA(cudaGraphAddKernelNode(&push, body, nullptr, 0, &p));
    void* args2[] = {&mg.state, &handle};
    p.func = mg.block == 128 ? (void*)k_ms_apply<128>
           : mg.block == 512 ? (void*)k_ms_apply<512> : (void*)k_ms_apply<256>;
    p.kernelParams = args2;
    HN_CUDA(cudaGraphAddKernelNode(&apply, body, &push, 1, &p));
    HN_CUDA(cudaGraphInstantiate(&mg.exec[part], graph, 0));
}

void build_ms_graph(hn_graph* g, MsGraph& mg) {
    const int nV = g->nV;
    // room for the graph to grow by a quarter before a rebuild
    const long long nchunk_cap = (g->nE + g->nE / 4) / kMsChunk + 1024;
    HN_CUDA(cudaMalloc((void**)&mg.state, sizeof(MsState)));
    HN_CUDA(cudaMallocHost((void**)&mg.h_state, sizeof(MsState)));
    HN_CUDA(cudaMalloc((void**)&mg.qbuf, sizeof(int32_t) * 2 * ((size_t)nV + 1)));
    HN_CUDA(cudaMalloc((void**)&mg.qbasebuf, sizeof(long long) * 2 * ((size_t)nV + 1)));
    HN_CUDA(cudaMalloc((void**)&mg.qoffbuf, sizeof(unsigned) * 2 * ((size_t)nV + 2)));
    HN_CUDA(cudaMalloc((void**)&mg.chunkbuf, sizeof(int32_t) * 2 * (size_t)nchunk_cap));
    HN_CUDA(cudaMalloc((void**)&mg.masks, sizeof(unsigned long long) * 4 * (size_t)nV));
    HN_CUDA(cudaMalloc((void**)&mg.touched, sizeof(int32_t) * ((size_t)nV + 1)));
    HN_CUDA(cudaMalloc((void**)&mg.stat, sizeof(unsigned long long) * 3 * kMaxSlots));
    HN_CUDA(cudaMallocHost((void**)&mg.h_stat, sizeof(unsigned long long) * 3 * kMaxSlots));
    mg.nV = nV;
    mg.nchunk_cap = nchunk_cap;

    build_ms_loop(g, mg, 0);
}

}  // namespace

void free_ms_graph(MsGraph* mg) {
    if (!mg) return;
    for (int i = 0; i < 2; i++) {
        if (mg->exec[i]) cudaGraphExecDestroy(mg->exec[i]);
        if (mg->graph[i]) cudaGraphDestroy(mg->graph[i]);
    }
    if (mg->state) cudaFree(mg->state);
    if (mg->h_state) cudaFreeHost(mg->h_state);
    if (mg->qbuf) cudaFree(mg->qbuf);
    if (mg->qbasebuf) cudaFree(mg->qbasebuf);
    if (mg->qoffbuf) cudaFree(mg->qoffbuf);
    if (mg->chunkbuf) cudaFree(mg->chunkbuf);
    if (mg->masks) cudaFree(mg->masks);
    if (mg->touched) cudaFree(mg->touched);
    if (mg->stat) cudaFree(mg->stat);
    if (mg->h_stat) cudaFreeHost(mg->h_stat);
    delete mg;
}

}  // namespace hn

using namespace hn;

extern "C" int hn_bfs_batch(hn_graph_t* g, const int32_t* sources, const int32_t* slots,
                            int32_t k, int32_t nslots, int32_t* dist, int mem,
                            hn_bfs_stats_t* slot_stats) {
    HN_API_BEGIN
    HN_REQUIRE(g && dist && (sources || k == 0), "null argument");
    HN_REQUIRE(nslots >= 1 && nslots <= kMaxSlots, "nslots must be in [1, 64]");
    HN_REQUIRE(k >= 0, "negative source count");
    HN_REQUIRE(slots || k <= nslots, "without slots, source j uses slot j (k <= nslots)");
    HN_REQUIRE(mem == HN_MEM_HOST || mem == HN_MEM_DEVICE, "bad memory kind");
    HN_REQUIRE(g->nV > 0, "empty graph");
    HN_REQUIRE(g->nE < 0xFFFFFFFFll, "batched BFS needs nE < 2^32");
    HandleUse use(g);
    HN_CUDA(cudaSetDevice(g->device));
    cudaStream_t s = g->stream;
    const int nV = g->nV;
    for (int j = 0; j < k; j++) {
        if (sources[j] < 0 || sources[j] >= nV) throw Error(HN_ERR_INVALID, "source outside [0, nV)");
        if (slots && (slots[j] < 0 || slots[j] >= nslots))
            throw Error(HN_ERR_INVALID, "slot outside [0, nslots)");
    }
    const int block = (int)knob(kKnobMsBlock);
    const unsigned grid = (unsigned)(g->info.sms * knob(kKnobMsCtasPerSm));
    if (g->ms && (g->ms->nV != nV || g->nE / kMsChunk + 4 > g->ms->nchunk_cap ||
                  g->ms->block != block || g->ms->grid != grid)) {
        HN_CUDA(cudaStreamSynchronize(s));
        free_ms_graph(g->ms);
        g->ms = nullptr;
    }
    if (!g->ms) {
        g->ms = new MsGraph();
        g->ms->block = block;
        g->ms->grid = grid;
        try {
            build_ms_graph(g, *g->ms);
        } catch (...) {
            free_ms_graph(g->ms);
            g->ms = nullptr;
            throw;
        }
    }
    MsGraph& mg = *g->ms;
    DevBuf<int32_t> d_src((size_t)k + 1, s), d_slot((size_t)k + 1, s), d_dist;
    if (k) {
        HN_CUDA(cudaMemcpyAsync(d_src.get(), sources, sizeof(int32_t) * k, cudaMemcpyHostToDevice, s));
        if (slots)
            HN_CUDA(cudaMemcpyAsync(d_slot.get(), slots, sizeof(int32_t) * k,
                                    cudaMemcpyHostToDevice, s));
    }
    int32_t* out = dist;
    if (mem == HN_MEM_HOST) {
        d_dist.alloc((size_t)nslots * nV, s);
        out = d_dist.get();
    }
    HN_CUDA(cudaStreamSynchronize(s));
    MsState& h = *mg.h_state;
    h = MsState{};
    h.nV = nV;
    h.nslots = nslots;
    h.vtab = g->vtab;
    h.pool = g->pool;
    h.q[0] = mg.qbuf;
    h.q[1] = mg.qbuf + nV + 1;
    h.qbase[0] = mg.qbasebuf;
    h.qbase[1] = mg.qbasebuf + nV + 1;
    h.qoff[0] = mg.qoffbuf;
    h.qoff[1] = mg.qoffbuf + nV + 2;
    h.chunk[0] = mg.chunkbuf;
    h.chunk[1] = mg.chunkbuf + mg.nchunk_cap;
    h.sn = (ulonglong2*)mg.masks;
    h.front[0] = mg.masks + 2 * (size_t)nV;
    h.front[1] = mg.masks + 3 * (size_t)nV;
    h.touched = mg.touched;
    h.dist = out;
    h.src = d_src.get();
    h.slot = slots ? d_slot.get() : nullptr;
    h.nsrc = k;
    h.stat = mg.stat;
    h.bottom_up = (int)knob(kKnobMsBottomUp);
    h.alpha = (int)knob(kKnobBfsDoAlpha);
    h.beta = (int)knob(kKnobBfsDoBeta);
    h.nE = h.open_edges = g->nE;
    h.check_min = knob(kKnobMsCheckMin);
    HN_CUDA(cudaMemcpyAsync(mg.state, &h, sizeof(MsState), cudaMemcpyHostToDevice, s));
    for (int part = 0; part < 2; part++) {   // at most twice: the answer is then known
        cudaEvent_t ev0 = nullptr;
        if (g_profiling) profile_begin(s, &ev0);
        HN_CUDA(cudaGraphLaunch(mg.exec[part], s));
        if (ev0) profile_end("k_ms_push+apply", s, ev0);
        count_launch(part == 0 ? 3 : 2);
        HN_CUDA(cudaMemcpyAsync(mg.h_stat, mg.stat, sizeof(unsigned long long) * 3 * kMaxSlots,
                                cudaMemcpyDeviceToHost, s));
        HN_CUDA(cudaMemcpyAsync(mg.h_state, mg.state, sizeof(MsState), cudaMemcpyDeviceToHost, s));
        HN_CUDA(cudaStreamSynchronize(s));
        if (!h.ask) break;
        if (!mg.exec[1]) build_ms_loop(g, mg, 1);
        check_symmetry(g, mg);
    }
    if (mem == HN_MEM_HOST) {
        HN_CUDA(cudaMemcpyAsync(dist, out, sizeof(int32_t) * (size_t)nslots * nV,
                                cudaMemcpyDeviceToHost, s));
        HN_CUDA(cudaStreamSynchronize(s));
    }
    if (slot_stats)
        for (int b = 0; b < nslots; b++) {
            slot_stats[b].levels =
                mg.h_stat[b] ? (int32_t)mg.h_stat[2 * kMaxSlots + b] + 1 : 0;
            slot_stats[b].pad = 0;
            slot_stats[b].visited = (int64_t)mg.h_stat[b];
            slot_stats[b].edges_scanned = (int64_t)mg.h_stat[kMaxSlots + b];
        }
    HN_API_END
}
