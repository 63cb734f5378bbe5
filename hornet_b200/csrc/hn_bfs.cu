// BFS TopDown (hornetsnest/src/Static/BreadthFirstSearch/TopDown.cu:49-106).
//
// Reference: per level, forAllEdges(queue, BFSOperator, BinarySearch) =
// computeWorkKernel + CUB scan + D2H total + binarySearchKernel with a
// non-atomic `dist[dst] == INF` test (duplicate enqueues possible), then a
// <<<1,1>>> swap kernel and another D2H (TwoLevelQueue.i.cuh:158-179): at
// least three host synchronisations per level.
//
// Here a whole BFS is ONE launch, without a host round trip between levels.
//   * Frontier entries are (vertex, adjacency base, edge offset).  The edge
//     offset is the exclusive prefix of the frontier's degrees; it comes out
//     of the enqueue itself: one 64-bit atomicAdd of (degree sum << 32 |
//     count) hands out the queue slots (low word) and the edge offsets (high
//     word) together, so offsets are ordered like slots and no scan runs.
//   * The frontier's edge space is cut into chunks of 2^cshift edges.  The
//     vertex that covers the first edge of each chunk records itself in
//     chunk[] when it is enqueued, so a chunk finds its vertex window with
//     two loads -- no search in global memory.  Only vertices with at least
//     one edge are queued, so a chunk of E edges spans at most E + 1 queue
//     entries.
//   * Visited-bitmap probes go through L1 (ld.ca): on power-law graphs most
//     edges point at a few hubs, and L2-only probes of their bitmap words
//     turn into a hot spot on a few L2 slices.  A stale L1 copy can only
//     miss bits set during this level (bits never clear), which costs an
//     extra atomicOr and never a wrong claim.  New vertices are claimed with
//     atomicOr on the bitmap (nV/8 bytes, L2-resident), so each vertex is
//     enqueued and its distance written exactly once.
//   * The last CTA of a level seals the next frontier; the loop also stops
//     after nV levels, so it always terminates.
//
// Two kernels share this frontier format (knob bfs.kernel):
//   * k_bfs_run (default): the whole BFS in one cooperative launch of one CTA
//     per SM (launch_run: fewer beside other BFS calls), with a grid barrier between levels (about 2 us; a kernel per
//     level in a WHILE node cost 8-15 us, whatever the level held).  A level
//     runs in one of four ways:
//       - up to 4,096 frontier edges: CTA 0 alone, level after level without
//         a grid barrier, frontier in shared memory (small_levels);
//       - up to one row of 32 edges per resident warp: thin_level;
//       - more: every WARP on its own, 256-edge chunks round-robin
//         (top_down_level).  It reads its window, loads its 8 x 32
//         neighbours lane-strided, probes and claims, and appends the claims
//         to a warp-private list in shared memory that is enqueued 32 or more
//         vertices at a time with one atomic;
//       - bottom_up_level, when directions may switch.
//     One B200, device time per source: scale 22 0.62 ms (0.65 with a kernel
//     per level), the direction-optimising form 0.28 (0.45), a 240,999-vertex
//     street grid of 654 levels 2.9 ms (11.8), a 4,096-vertex R-MAT graph
//     50 us (75).
//   * k_bfs_level (bfs.kernel = 0): a WHILE node around a kernel per level, a
//     CTA of 128 threads per 1024-edge chunk, with the window staged in
//     shared memory and a CTA-wide enqueue (one atomic per chunk).
// Distances equal the reference's: level-synchronous, INF = INT32_MAX.
//
// hn_bfs_do runs the same kernel with levels that may run bottom-up (Beamer's
// direction-optimising BFS, the counterpart of hornetsnest's BottomUpBFS,
// src/Static/BottomUpBreadthFirstSearch/BottomUpBFS.cu); on a graph that
// stores every edge both ways distances are identical, and fewer edges are
// read.
#include <algorithm>
#include <climits>

#include "hn_graph.cuh"
#include "hn_gridsync.cuh"

namespace hn {

constexpr int kBfsBlock = 128;
constexpr int kIpt = 8;                          // edges per thread per chunk
constexpr int kChunk = kBfsBlock * kIpt;         // edges per CTA chunk (k_bfs_level)
constexpr int kChunkShiftCta = 10;               // log2(kChunk)
constexpr int kWIpt = 8;                         // edges per lane per warp chunk
constexpr int kWChunk = 32 * kWIpt;              // edges per warp chunk
constexpr int kChunkShiftWarp = 8;               // log2(kWChunk)
constexpr int kWList = kWChunk + 32;             // claim list capacity per warp
static_assert(kChunk == 1 << kChunkShiftCta && kWChunk == 1 << kChunkShiftWarp, "chunk sizes");

constexpr int kTraceLevels = 32;

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct BfsState {
    unsigned long long cnt[3];   // frontier counters: (edge total << 32) | size
    int level;                   // distance given to vertices found now
    unsigned ticket;             // CTAs finished with the current level
    long long visited;
    long long scanned;
    int src;
    int nV;
    int32_t* dist;
    const VRec* vtab;
    const int32_t* pool;
    int32_t* q[2];               // frontier vertices
    long long* qbase[2];         // their adjacency base in the pool
    unsigned* qoff[2];           // exclusive degree prefix (edge offset)
    int32_t* chunk[2];           // queue slot covering each chunk's first edge
    unsigned* bitmap;            // visited bits
    int mode;                    // direction-optimising: 0 top-down, 1 bottom-up
    int pad;
    long long m_total;           // edges of the graph
    long long edges_visited;     // sum of degrees of vertices reached so far
    int alpha;                   // direction-optimising switch thresholds
    int beta;
    int dynamic_chunks;          // 1: CTAs take chunks from next_chunk
    unsigned next_chunk;         // chunk counter of the current level
    int warp_strided;            // 1: a warp's edges are lane-strided (coalesced loads)
    int cont;                    // 1 while another level follows (host-driven loop)
    int host_driven;             // 1: no conditional node (levels launched by the host)
    int cshift;                  // log2 of the chunk size of chunk[]
    // level trace: global timer (ns) at the start and at the end of each of
    // the first kTraceLevels levels, and the frontier edges each one scanned
    unsigned long long t_start;
    unsigned long long t_end[kTraceLevels];
    unsigned long long lvl_edges[kTraceLevels];
};

// What a finished BFS hands to the host (pinned; written by k_bfs_run).
struct BfsOut {
    int level;                   // levels run + 1
    int done;                    // 0: stopped at max_levels, more to do
    int error;                   // HN_ERR_TIMEOUT when a grid wait gave up
    int pad;
    long long visited;
    long long scanned;
    unsigned long long t_start;  // level trace, as in BfsState
    unsigned long long t_end[kTraceLevels];
    unsigned long long lvl_edges[kTraceLevels];
};

struct BfsCtl;

struct BfsGraph {
    int nV = -1;
    long long nchunk_cap = 0;
    char* mem = nullptr;            // one device allocation holding all of the arrays below
    long long* qbasebuf = nullptr;
    unsigned* qoffbuf = nullptr;
    int32_t* chunkbuf = nullptr;
    unsigned* bitmap = nullptr;
    unsigned grid = 0;                              // level-kernel CTAs
    unsigned threads = 0;                           // threads per CTA
    int kernel = -1;                                // bfs.kernel
    // k_bfs_run
    BfsCtl* ctl = nullptr;          // device
    unsigned* fbits = nullptr;      // two frontier bitmaps
    // k_bfs_level
    BfsState* state = nullptr;      // device
    BfsState* h_state = nullptr;    // pinned
    int32_t* qbuf = nullptr;
    cudaGraph_t graph[2] = {nullptr, nullptr};      // [0] top-down, [1] direction-optimising
    cudaGraphExec_t exec[2] = {nullptr, nullptr};
    // multi-source calls: pinned per-source results (k_bfs_run) or states
    // (k_bfs_level: the next source's is staged while the previous BFS runs),
    // a copy stream and events so a host-bound distance array is copied out
    // while the next BFS runs
    static constexpr int kRing = 64;
    BfsOut* h_out = nullptr;                        // pinned, kRing entries
    BfsState* h_ring = nullptr;                     // pinned, kRing entries (k_bfs_level)
    cudaStream_t copy = nullptr;
    cudaEvent_t done[2] = {nullptr, nullptr};       // BFS into buffer b finished
    cudaEvent_t copied[2] = {nullptr, nullptr};     // buffer b copied to the host
    BfsOut last = {};                               // result of the latest BFS
    bool have_last = false;
};

namespace {

// Record queue slot `pos` as the owner of every chunk (2^cs edges) whose
// first edge lies in [off, off + d).
__device__ __forceinline__ void mark_chunks(int32_t* chunk, unsigned off, unsigned d, int pos,
                                            int cs) {
    unsigned c0 = (off + (1u << cs) - 1) >> cs;
    unsigned c1 = (off + d - 1) >> cs;
    for (unsigned c = c0; c <= c1; c++) chunk[c] = pos;
}

__global__ void k_bfs3_init(BfsState* st) {
    const int nV = st->nV;
    const int src = st->src;
    int32_t* dist = st->dist;
    unsigned* bm = st->bitmap;
    long long nwords = ((long long)nV + 31) / 32;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nV;
         i += (long long)gridDim.x * blockDim.x) {
        dist[i] = i == src ? 0 : kInf;
        if (i < nwords) bm[i] = (i == src / 32) ? (1u << (src & 31)) : 0u;
    }
    VRec r = st->vtab[src];
    unsigned d = (unsigned)r.deg;
    // chunk marks of a high-degree source are spread over the grid
    if (d > 0) {
        unsigned nc = ((d - 1) >> st->cshift) + 1;
        for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < nc;
             c += (long long)gridDim.x * blockDim.x)
            st->chunk[0][c] = 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->q[0][0] = src;
        st->qbase[0][0] = r.off;
        st->qoff[0][0] = 0;
        st->qoff[0][d > 0 ? 1 : 0] = d;
        st->cnt[0] = d > 0 ? (((unsigned long long)d << 32) | 1ull) : 0ull;
        st->cnt[1] = 0;
        st->cnt[2] = 0;
        st->level = 1;
        st->ticket = 0;
        st->visited = 1;
        st->scanned = 0;
        st->mode = 0;
        st->edges_visited = d;
        st->t_start = global_ns();
    }
}

// Per-level shared memory of the level kernel.
struct BfsSmem {
    unsigned start[kChunk + 2];   // window edge offsets (+ end)
    long long base[kChunk + 1];   // pool index = base + edge
    int claimed[kChunk];          // vertices claimed in this chunk
    int nclaimed;
    int nw;
    unsigned next;                // this CTA's next chunk
    unsigned long long wsum[kBfsBlock / 32];
    unsigned long long cbase;
};

// CTA-wide enqueue of the chunk's claimed vertices.  The claims are first
// gathered into shared memory (one shared atomic per warp), then each thread
// takes an equal contiguous share of them: distance written, and vertices
// with edges appended to the next frontier with their adjacency base and
// edge offset; ONE atomic per call reserves both the queue slots and the
// edge range.  Holding no per-claim arrays keeps the kernel's register
// count, and so its residency, down.  Must be called by all threads.
__device__ __forceinline__ void bfs_enqueue(BfsSmem& sm, const int (&w)[kIpt],
                                            const bool (&claim)[kIpt], int level,
                                            const VRec* __restrict__ vtab, int32_t* dist,
                                            unsigned long long* cout, int32_t* nqv,
                                            long long* nqbase, unsigned* nqoff, int32_t* nchunk,
                                            int cs, int& found) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) sm.nclaimed = 0;
    __syncthreads();
    {
        int mine = 0;
#pragma unroll
        for (int k = 0; k < kIpt; k++) mine += claim[k] ? 1 : 0;
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += x;
        }
        const int wtot = __shfl_sync(0xFFFFFFFFu, incl, 31);
        int wbase = 0;
        if (lane == 31 && wtot) wbase = atomicAdd(&sm.nclaimed, wtot);
        wbase = __shfl_sync(0xFFFFFFFFu, wbase, 31);
        int at = wbase + incl - mine;
#pragma unroll
        for (int k = 0; k < kIpt; k++)
            if (claim[k]) sm.claimed[at++] = w[k];
    }
    __syncthreads();
    const int n = sm.nclaimed;
    if (n == 0) return;   // uniform: every thread read the same count
    const int per = (n + kBfsBlock - 1) / kBfsBlock;
    const int i0 = threadIdx.x * per;
    const int i1 = i0 + per < n ? i0 + per : n;
    unsigned long long mine = 0;   // (degree sum << 32) | queued count
    for (int i = i0; i < i1; i++) {
        const int v = sm.claimed[i];
        const int d = vtab[v].deg;
        dist[v] = level;
        found++;
        if (d) mine += ((unsigned long long)d << 32) | 1ull;
    }
    unsigned long long incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long x = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += x;
    }
    const int warp = threadIdx.x >> 5;
    if (lane == 31) sm.wsum[warp] = incl;
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned long long v = threadIdx.x < kBfsBlock / 32 ? sm.wsum[threadIdx.x] : 0ull;
        unsigned long long vi = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned long long x = __shfl_up_sync(0xFFFFFFFFu, vi, o);
            if (lane >= o) vi += x;
        }
        if (threadIdx.x < kBfsBlock / 32) sm.wsum[threadIdx.x] = vi - v;   // exclusive
        unsigned long long tot = __shfl_sync(0xFFFFFFFFu, vi, 31);
        if (threadIdx.x == 0) sm.cbase = tot ? atomicAdd(cout, tot) : 0ull;
    }
    __syncthreads();
    unsigned long long at = sm.cbase + sm.wsum[warp] + (incl - mine);
    int pos = (int)(at & 0xFFFFFFFFull);
    unsigned off = (unsigned)(at >> 32);
    for (int i = i0; i < i1; i++) {
        const int v = sm.claimed[i];
        const VRec r = vtab[v];   // second read of the record: an L1 hit
        if (r.deg) {
            nqv[pos] = v;
            nqbase[pos] = r.off;
            nqoff[pos] = off;
            mark_chunks(nchunk, off, (unsigned)r.deg, pos, cs);
            pos++;
            off += (unsigned)r.deg;
        }
    }
    __syncthreads();
}

// End of a level, called by every thread of every CTA: the visited count
// (one atomic per warp), then the last CTA seals the next frontier, picks the
// next direction and decides whether to loop.
template <bool DO>
__device__ __forceinline__ void bfs_level_end(BfsState* st, cudaGraphConditionalHandle cond,
                                              int found, int level, int nq, unsigned total,
                                              unsigned long long* cout, unsigned* nqoff) {
    const int lane = threadIdx.x & 31;
    for (int o = 16; o; o >>= 1) found += __shfl_down_sync(0xFFFFFFFFu, found, o);
    if (lane == 0 && found) atomicAdd((unsigned long long*)&st->visited, (unsigned long long)found);
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned tk = atomicAdd(&st->ticket, 1u);
        if (tk == gridDim.x - 1) {
            __threadfence();
            unsigned long long cn = atomicAdd(cout, 0ull);
            unsigned nn = (unsigned)(cn & 0xFFFFFFFFull);
            unsigned long long mf = cn >> 32;
            nqoff[nn] = (unsigned)mf;
            st->ticket = 0;
            st->next_chunk = 0;
            st->scanned += total;
            if (level <= kTraceLevels) {
                st->t_end[level - 1] = global_ns();
                st->lvl_edges[level - 1] = total;
            }
            st->level = level + 1;
            if (DO) {
                // Beamer's switch: to bottom-up when the next frontier's edges
                // exceed 1/alpha of the unexplored edges (alpha = 4 by
                // default), back to top-down when the frontier falls below
                // nV/beta vertices (beta = 24) and is shrinking
                st->edges_visited += (long long)mf;
                long long mu = st->m_total - st->edges_visited;
                if (st->mode == 0) {
                    if ((long long)mf * st->alpha > mu) st->mode = 1;
                } else {
                    if ((long long)nn * st->beta < st->nV && nn < (unsigned)nq) st->mode = 0;
                }
            }
            const unsigned more = (nn > 0 && level < st->nV) ? 1u : 0u;
            st->cont = (int)more;
            if (!st->host_driven) cudaGraphSetConditional(cond, more);
        }
    }
}

// ---------------------------------------------------------------------------
// k_bfs_run: a whole BFS in one cooperative launch (bfs.kernel = 1).
// ---------------------------------------------------------------------------

}  // namespace

// Device state shared by the CTAs of a launch (and by the launches of one
// BFS when the host drives its levels).
struct BfsCtl {
    unsigned long long cout;     // next frontier: (edge total << 32) | size
    unsigned long long cin;      // current frontier, sealed
    GridBar bar;                 // beat: CTA 0's small levels, while the others wait
    int level;                   // distance given to vertices found now
    int mode;                    // 0 top-down, 1 bottom-up
    int cur;                     // queue buffer of the current frontier
    int fcur;                    // frontier bitmap of the current (bottom-up) frontier
    int marks;                   // 1: chunk[] of the current frontier is still to be written
    int done;
    int left;                    // levels this launch may still run
    long long visited;
    long long scanned;
    long long edges_visited;     // sum of degrees of vertices reached so far
    // CTA 0's state after its small levels; the next barrier's seal takes it
    // over (other CTAs may still be reading the fields above)
    unsigned long long s_cin;
    int s_level, s_mode, s_marks, s_done, s_left, s_pad;
    long long s_scanned, s_edges;
};

namespace {

struct BfsArgs {
    BfsCtl* ctl;
    BfsOut* out;
    const VRec* vtab;
    const int32_t* pool;
    int32_t* dist;
    unsigned* bitmap;            // visited
    unsigned* fbits[2];          // frontier bitmaps (bottom-up levels)
    long long* qbase[2];         // adjacency base of each frontier vertex
    unsigned* qoff[2];           // exclusive degree prefix
    int32_t* chunk[2];           // queue slot covering each chunk's first edge
    long long m_total;
    int nV, src;
    int alpha, beta;             // direction switch (DO)
    // (in one word: with eight bytes more of arguments k_bfs_run spilled twice as
    // much, and 16 traversals of scale 22 took 10.1 ms instead of 9.7)
    unsigned first : 1;          // 1: a new BFS (0: the next levels of one)
    unsigned wait_polls : 31;    // limit of a wait at the grid barrier
    int max_levels;
};

// Warp-private shared memory of the grid-wide levels.
struct WarpSmem {
    long long base[kWList];        // window: pool index = base + edge (large windows);
                                   // flush: adjacency base of each listed vertex
    unsigned start[kWList];        // window edge offsets (+ end); flush: degrees
    int list[kWList];              // claimed vertices not yet enqueued
};

// Frontiers of at most kSmallEdges edges are expanded by CTA 0 alone, in
// shared memory: a grid barrier costs about as much as four edges a thread,
// and a level of a long, thin frontier is one chain of dependent loads
// either way.
constexpr int kSmallEdges = 4096;
struct SmallSmem {
    long long base[2][kSmallEdges];     // pool index = base + edge
    unsigned off[2][kSmallEdges + 1];   // edge offsets (+ end)
    unsigned long long wsum[32];
    unsigned long long next;            // next frontier so far
};

// Per-CTA copy of the level's state, and where its claims go (the enqueue is
// rare next to the edge loop, so these do not hold registers there).
struct LevelSmem {
    BfsArgs a;
    unsigned long long cin;
    int level, mode, cur, fcur, marks, done, error;
    unsigned gen;                // barrier generation (thread 0's)
    const VRec* vtab;
    int32_t* dist;
    unsigned long long* cout;
    long long* nqbase;
    unsigned* nqoff;
    int32_t* nchunk;
};

// 768 threads an SM (80 registers): top_down_level spills at 64 (1024
// threads; its largest level at scale 22: 540-640 us against 375-425).
constexpr int kRunThreads = 768;
constexpr size_t kLevelSmem = (sizeof(LevelSmem) + 15) & ~(size_t)15;
constexpr size_t kRunSmem =
    kLevelSmem + (sizeof(WarpSmem) * (kRunThreads / 32) > sizeof(SmallSmem)
                      ? sizeof(WarpSmem) * (kRunThreads / 32) : sizeof(SmallSmem));

// Dynamic shared memory of k_bfs_run: the level's state, then either the
// warps' or CTA 0's small-level buffers.  The rarer phases of a level are
// functions of their own (not inlined, so that the edge loop of
// top_down_level keeps the registers); all reach shared memory through these,
// not through arguments, which would make every access a generic one.
extern __shared__ __align__(16) unsigned char s_run[];
__device__ __forceinline__ LevelSmem& level_smem() { return *reinterpret_cast<LevelSmem*>(s_run); }
__device__ __forceinline__ WarpSmem& warp_smem() {
    return reinterpret_cast<WarpSmem*>(s_run + kLevelSmem)[threadIdx.x >> 5];
}
__device__ __forceinline__ SmallSmem& small_smem() {
    return *reinterpret_cast<SmallSmem*>(s_run + kLevelSmem);
}
__device__ __forceinline__ unsigned grid_warp() {
    return blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
}
__device__ __forceinline__ unsigned grid_warps() { return gridDim.x * (blockDim.x >> 5); }

// Enqueue all n vertices of the warp's claim list in one pass: every lane
// reads the records of up to ceil(n / 32) listed vertices (loads issued
// together) into the warp's shared memory and writes their distances (DIST),
// then one warp scan and ONE 64-bit atomicAdd reserve the queue slots and the
// edge range of all of them, and each lane writes its consecutive share of
// queue entries.  A vertex that spans many chunks has its chunk marks
// written by the whole warp.  Called by all 32 lanes with the same n.
template <bool DIST>
__device__ __forceinline__ void warp_flush(WarpSmem& sm, int n, const LevelSmem& lo, int& found) {
    const int lane = threadIdx.x & 31;
    const VRec* __restrict__ vtab = lo.vtab;
    int32_t* dist = lo.dist;
    const int level = lo.level;
    const unsigned kFull = 0xFFFFFFFFu;
    // records of the listed vertices, four loads in flight per lane
    for (int i0 = 0; i0 < n; i0 += 128) {
        VRec r[4];
        int v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = i0 + u * 32 + lane;
            v[u] = i < n ? sm.list[i] : -1;
            if (v[u] >= 0) r[u] = vtab[v[u]];
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int i = i0 + u * 32 + lane;
            if (v[u] >= 0) {
                if (DIST) {
                    dist[v[u]] = level;
                    found++;
                }
                sm.base[i] = r[u].off;
                sm.start[i] = (unsigned)r[u].deg;
            }
        }
    }
    __syncwarp();
    // lane L owns list entries [L * per, L * per + per)
    const int per = (n + 31) >> 5;
    const int i0 = lane * per;
    const int i1 = i0 + per < n ? i0 + per : n;
    unsigned long long mine = 0;   // (degree sum << 32) | vertices with edges
    for (int i = i0; i < i1; i++) {
        const unsigned d = sm.start[i];
        if (d) mine += ((unsigned long long)d << 32) | 1ull;
    }
    unsigned long long incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        unsigned long long x = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += x;
    }
    unsigned long long base = 0;
    if (lane == 31 && incl) base = atomicAdd(lo.cout, incl);
    base = __shfl_sync(kFull, base, 31);
    unsigned long long at = base + incl - mine;
    bool has_big = false;
    long long* nqbase = lo.nqbase;
    unsigned* nqoff = lo.nqoff;
    int32_t* nchunk = lo.nchunk;
    for (int i = i0; i < i1; i++) {
        const unsigned d = sm.start[i];
        if (!d) continue;
        const int pos = (int)(at & 0xFFFFFFFFull);
        const unsigned off = (unsigned)(at >> 32);
        nqbase[pos] = sm.base[i];
        nqoff[pos] = off;
        const unsigned c0 = (off + kWChunk - 1) >> kChunkShiftWarp;
        const unsigned c1 = (off + d - 1) >> kChunkShiftWarp;
        if (c1 < c0 + 8) {
            for (unsigned c = c0; c <= c1; c++) nchunk[c] = pos;
        } else {
            // marked below by the whole warp: keep its (slot, offset)
            sm.base[i] = (long long)at;
            sm.start[i] = d | 0x80000000u;
            has_big = true;
        }
        at += ((unsigned long long)d << 32) | 1ull;
    }
    // vertices spanning many chunks: their chunk marks written by the warp
    unsigned bigm = __ballot_sync(kFull, has_big);
    __syncwarp();
    while (bigm) {
        const int src = __ffs(bigm) - 1;
        bigm &= bigm - 1;
        const int j0 = src * per;
        const int j1 = j0 + per < n ? j0 + per : n;
        for (int i = j0; i < j1; i++) {
            const unsigned f = sm.start[i];
            if (!(f & 0x80000000u)) continue;
            const unsigned d = f & 0x7FFFFFFFu;
            const unsigned long long a2 = (unsigned long long)sm.base[i];
            const int pos = (int)(a2 & 0xFFFFFFFFull);
            const unsigned off = (unsigned)(a2 >> 32);
            const unsigned c0 = (off + kWChunk - 1) >> kChunkShiftWarp;
            const unsigned c1 = (off + d - 1) >> kChunkShiftWarp;
            for (unsigned c = c0 + lane; c <= c1; c += 32) nchunk[c] = pos;
        }
    }
    __syncwarp();
}

// Append the lanes' claimed vertices (bit k of `claim` set: w[k] claimed) to
// the warp list and flush it once it holds 32 or more.
template <bool DIST, int N>
__device__ __forceinline__ void warp_claims(WarpSmem& sm, int& nlist, const int (&w)[N],
                                            unsigned claim, const LevelSmem& lo, int& found) {
    const int lane = threadIdx.x & 31;
    const unsigned kFull = 0xFFFFFFFFu;
    if (!__any_sync(kFull, claim != 0u)) return;
    const int mine = __popc(claim);
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int x = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += x;
    }
    const int tot = __shfl_sync(kFull, incl, 31);
    if (tot == 0) return;
    int at = nlist + incl - mine;
#pragma unroll
    for (int k = 0; k < N; k++)
        if (claim >> k & 1u) sm.list[at++] = w[k];
    nlist += tot;
    __syncwarp();
    if (nlist >= 32) {
        warp_flush<DIST>(sm, nlist, lo, found);
        nlist = 0;
    }
}

// A grid-wide top-down level of one warp: 256-edge chunks round-robin.  A
// chunk's vertex window comes from chunk[] with two loads; windows of at most
// 32 vertices stay in registers, where a lane finds the vertex of each of its
// edges with one OR-reduction, one ballot and one shuffle.  Each load
// instruction reads 32 consecutive edges.  (The queue arrays change during
// the launch: they are read with ordinary loads, after the grid barrier's
// fence, never through the read-only path.)
__device__ __forceinline__ int top_down_level() {
    WarpSmem& sm = warp_smem();
    const LevelSmem& lo = level_smem();
    const BfsArgs& a = lo.a;
    const unsigned gw = grid_warp(), nwarps = grid_warps();
    int found = 0;
    const unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const int nq = (int)(lo.cin & 0xFFFFFFFFull);
    const unsigned total = (unsigned)(lo.cin >> 32);
    const long long* qbase = a.qbase[lo.cur];
    const unsigned* qoff = a.qoff[lo.cur];
    const int32_t* chunk = a.chunk[lo.cur];
    const int32_t* __restrict__ pool = a.pool;
    unsigned* bm = a.bitmap;
    const unsigned nchunks = (total + kWChunk - 1) >> kChunkShiftWarp;
    int nlist = 0;
    // A chunk's window: its first queue entry s0 and its size nw; with at
    // most 32 entries, lane j holds entry s0 + j (start sj, base bj).
    int s0 = 0, nw = 0;
    unsigned sj = 0xFFFFFFFFu;
    long long bj = 0;
    if (gw < nchunks) {
        s0 = chunk[gw];
        nw = (gw + 1 < nchunks ? chunk[gw + 1] : nq - 1) - s0 + 1;
        if (nw <= 32 && lane < nw) {
            sj = qoff[s0 + lane];
            bj = qbase[s0 + lane] - (long long)sj;
        }
    }
    // The next chunk's window is read while this chunk's neighbour loads are
    // in flight, so a chunk waits on three round trips (neighbours, bitmap,
    // claims), not five.
    for (unsigned c = gw; c < nchunks; c += nwarps) {
        const unsigned cn = c + nwarps;
        int ns0 = 0, ns1 = -1;
        if (cn < nchunks) {
            ns0 = chunk[cn];
            ns1 = cn + 1 < nchunks ? chunk[cn + 1] : nq - 1;   // inclusive
        }
        const unsigned e0 = c << kChunkShiftWarp;
        const unsigned e1 = e0 + kWChunk < total ? e0 + kWChunk : total;
        int w[kWIpt];   // the chunk's neighbours, lane-strided (-1 past the frontier's end)
#pragma unroll
        for (int k = 0; k < kWIpt; k++) w[k] = -1;
        if (nw == 1) {
            // one vertex covers the chunk (hubs): no owner search
            const long long b = __shfl_sync(kFull, bj, 0);
#pragma unroll
            for (int k = 0; k < kWIpt; k++) {
                const unsigned e = e0 + 32u * k + lane;
                if (e < e1) w[k] = __ldg(pool + b + e);
            }
        } else if (nw <= 32) {
            // the vertex of edge e is the last entry starting at or before
            // e: entries started before the row (ballot) plus starts inside
            // the row up to this lane (OR-reduced bits)
#pragma unroll
            for (int k = 0; k < kWIpt; k++) {
                const unsigned rs = e0 + 32u * k;
                const unsigned rel = sj - rs;   // wraps for entries before the row
                const unsigned bits = __reduce_or_sync(kFull, lane < nw && sj >= rs && rel < 32u
                                                                  ? 1u << rel : 0u);
                const int before = __popc(__ballot_sync(kFull, lane < nw && sj < rs));
                const int j = before - 1 + __popc(bits & (kFull >> (31 - lane)));
                const long long b = __shfl_sync(kFull, bj, j & 31);
                const unsigned e = rs + lane;
                if (e < e1) w[k] = __ldg(pool + b + e);
            }
        } else {
            // larger window: staged in the warp's shared memory, one search
            // per lane over 8 consecutive edges
            for (int j = lane; j <= nw; j += 32) {
                const unsigned so = qoff[s0 + j];   // qoff[nq] is the sealed total
                sm.start[j] = so;
                if (j < nw) sm.base[j] = qbase[s0 + j] - (long long)so;
            }
            __syncwarp();
            const unsigned x = e0 + lane * kWIpt;
            int lo2 = 0, hi = nw;                   // last j with start[j] <= x
            while (hi - lo2 > 1) {
                const int mid = (lo2 + hi) >> 1;
                if (sm.start[mid] <= x) lo2 = mid; else hi = mid;
            }
            int j = lo2;
#pragma unroll
            for (int k = 0; k < kWIpt; k++) {
                const unsigned e = x + k;
                if (e < e1) {
                    while (sm.start[j + 1] <= e) j++;
                    w[k] = __ldg(pool + sm.base[j] + e);
                }
            }
            __syncwarp();
        }
        // the next chunk's register window
        s0 = ns0;
        nw = ns1 - ns0 + 1;
        sj = 0xFFFFFFFFu;
        bj = 0;
        if (nw <= 32 && lane < nw) {
            sj = qoff[s0 + lane];
            bj = qbase[s0 + lane] - (long long)sj;
        }
        unsigned word[kWIpt];
#pragma unroll
        for (int k = 0; k < kWIpt; k++)
            word[k] = w[k] >= 0 ? __ldca(bm + (w[k] >> 5)) : 0xFFFFFFFFu;
        unsigned claim = 0;
#pragma unroll
        for (int k = 0; k < kWIpt; k++) {
            if (w[k] >= 0 && !(word[k] & (1u << (w[k] & 31)))) {
                const unsigned bit = 1u << (w[k] & 31);
                if (!(atomicOr(bm + (w[k] >> 5), bit) & bit)) claim |= 1u << k;
            }
        }
        warp_claims<true>(sm, nlist, w, claim, lo, found);
    }
    if (nlist > 0) warp_flush<true>(sm, nlist, lo, found);
    return found;
}

// A grid-wide top-down level with at most one row of 32 edges per resident
// warp: the rows of a chunk go to different warps, so the level is one chain
// of loads, and claims are enqueued at once.  The records of all neighbours
// are read with the bitmap probes (one round trip less than after the
// claims).  A row finds its queue entries by search, so thin levels read no
// chunk marks, and leave those of the next frontier to the grid (ctl->marks):
// a few warps would otherwise write the marks of all the hubs they reach.
__device__ __noinline__ int thin_level() {
    const LevelSmem& lo = level_smem();
    const BfsArgs& a = lo.a;
    const unsigned gw = grid_warp();
    const unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const int nq = (int)(lo.cin & 0xFFFFFFFFull);
    const unsigned total = (unsigned)(lo.cin >> 32);
    const unsigned row = gw * 32u;
    if (row >= total) return 0;
    const long long* qbase = a.qbase[lo.cur];
    const unsigned* qoff = a.qoff[lo.cur];
    // last entry starting at or before the row, 32 probes a step
    int s0 = 0;
    for (int n = nq; n > 1;) {
        const int step = (n + 31) / 32;
        const int i = s0 + lane * step;
        const bool le = lane * step < n && __ldcg(qoff + i) <= row;
        const int j = __popc(__ballot_sync(kFull, le)) - 1;   // entry s0 starts at or before it
        s0 += j * step;
        n = n - j * step < step ? n - j * step : step;
    }
    // the row's 32 edges meet at most 32 entries: lane j holds entry s0 + j
    const bool in = s0 + lane < nq;
    const unsigned sj = in ? __ldcg(qoff + s0 + lane) : 0xFFFFFFFFu;
    const long long bj = in ? __ldcg(qbase + s0 + lane) - (long long)sj : 0;
    const unsigned rel = sj - row;
    const unsigned bits = __reduce_or_sync(kFull, in && sj > row && rel < 32u ? 1u << rel : 0u);
    const int owner = __popc(bits & (kFull >> (31 - lane)));
    const long long b = __shfl_sync(kFull, bj, owner);
    const unsigned e = row + lane;
    const int w = e < total ? __ldg(a.pool + b + e) : -1;
    bool claim = false;
    VRec r;
    r.off = 0;
    r.deg = r.cap = 0;
    if (w >= 0) {
        const unsigned bit = 1u << (w & 31);
        const unsigned word = __ldca(a.bitmap + (w >> 5));
        r = a.vtab[w];
        if (!(word & bit)) claim = !(atomicOr(a.bitmap + (w >> 5), bit) & bit);
    }
    if (claim) lo.dist[w] = lo.level;
    const unsigned long long mine =
        claim && r.deg ? ((unsigned long long)(unsigned)r.deg << 32) | 1ull : 0ull;
    unsigned long long incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long x = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += x;
    }
    unsigned long long base = 0;
    if (lane == 31 && incl) base = atomicAdd(lo.cout, incl);
    const unsigned long long at = __shfl_sync(kFull, base, 31) + incl - mine;
    if (mine) {
        const int pos = (int)(at & 0xFFFFFFFFull);
        lo.nqbase[pos] = r.off;
        lo.nqoff[pos] = (unsigned)(at >> 32);
    }
    return claim ? 1 : 0;
}

// Frontier bitmap of the vertices at distance level - 1 (top-down ->
// bottom-up).  A warp takes 256 vertices (eight words).
__device__ __noinline__ void frontier_bits() {
    const LevelSmem& lo = level_smem();
    const int32_t* dist = lo.a.dist;
    unsigned* fb = lo.a.fbits[0];
    const int nV = lo.a.nV, level = lo.level;
    const unsigned gw = grid_warp(), nwarps = grid_warps();
    const int lane = threadIdx.x & 31;
    const unsigned units = ((unsigned)nV + kWChunk - 1) >> kChunkShiftWarp;
    const unsigned nwords = ((unsigned)nV + 31) / 32;
    for (unsigned c = gw; c < units; c += nwarps) {
        int d[kWIpt];
        unsigned mine = 0;
#pragma unroll
        for (int k = 0; k < kWIpt; k++) {
            const long long v = ((long long)c << kChunkShiftWarp) + 32 * k + lane;
            d[k] = v < nV ? __ldcg(dist + v) : -1;
        }
#pragma unroll
        for (int k = 0; k < kWIpt; k++) {
            const unsigned b = __ballot_sync(0xFFFFFFFFu, d[k] == level - 1);
            if (lane == k) mine = b;
        }
        if (lane < kWIpt && c * kWIpt + lane < nwords) fb[c * kWIpt + lane] = mine;
    }
}

// Bottom-up level: every unvisited vertex looks for a neighbour on the
// frontier (bitmap fb: nV / 8 bytes, against 4 nV for distances) and stops at
// the first (Beamer, Asanovic & Patterson, "Direction-Optimizing
// Breadth-First Search", SC 2012).  A lane reads the first kBuLane neighbours
// of its vertex itself, four at a time; a longer list without a hit is then
// read by the whole warp, 64 neighbours a step, so a hub off the frontier
// costs its warp deg / 64 steps (four lists at a time by eight lanes each
// measured 5 % slower).  A warp owns whole words of the visited and
// next-frontier bitmaps, so both are written with plain stores.
constexpr int kBuLane = 16;
// Entries of long lists that a warp reads between two signs of progress (2,048
// steps, 1.2 ms): its share of a level has no bound but the edge count.
constexpr int kBuBeat = 1 << 17;

__device__ __noinline__ int bottom_up_level() {
    const LevelSmem& lo = level_smem();
    const BfsArgs& a = lo.a;
    const int level = lo.level;
    const unsigned* fb = a.fbits[lo.fcur & 1];
    unsigned* nfb = a.fbits[(lo.fcur & 1) ^ 1];
    unsigned long long* cout = lo.cout;
    const unsigned gw = grid_warp(), nwarps = grid_warps();
    int found = 0;
    const unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31;
    const int nV = a.nV;
    const VRec* __restrict__ vtab = a.vtab;
    const int32_t* __restrict__ pool = a.pool;
    unsigned* bm = a.bitmap;
    int32_t* const dist = a.dist;
    const unsigned units = ((unsigned)nV + kWChunk - 1) >> kChunkShiftWarp;
    const unsigned nwords = ((unsigned)nV + 31) / 32;
    unsigned long long queued = 0;   // (degree sum << 32) | vertices with edges
    int beat = 0;                    // entries of long lists since the last sign of progress
    for (unsigned c = gw; c < units; c += nwarps) {
        const unsigned word = c * kWIpt + lane;
        const bool own = lane < kWIpt && word < nwords;
        const unsigned vis = own ? __ldcg(bm + word) : kFull;
        unsigned fresh = 0;
        auto record = [&](int k) {   // of this lane's vertex of word k, empty when visited
            const unsigned un = ~__shfl_sync(kFull, vis, k);
            const long long v = ((long long)c << kChunkShiftWarp) + 32 * k + lane;
            VRec r;
            r.off = 0;
            r.deg = r.cap = 0;
            if ((un >> lane & 1u) && v < nV) r = vtab[v];
            return r;
        };
        VRec rn = record(0);
#pragma unroll 1
        for (int k = 0; k < kWIpt; k++) {
            const VRec r = rn;
            if (k + 1 < kWIpt) rn = record(k + 1);   // in flight while word k is processed
            if (!__any_sync(kFull, r.deg > 0)) continue;
            const long long v = ((long long)c << kChunkShiftWarp) + 32 * k + lane;
            bool hit = false;
            const int32_t* nb = pool + r.off;
            const int mine = r.deg < kBuLane ? r.deg : kBuLane;
            for (int e = 0; e < mine && !hit; e += 4) {
                int4 n4;   // blocks of capacity >= 4 are 16-byte aligned and whole
                if (r.cap >= 4) n4 = __ldg(reinterpret_cast<const int4*>(nb + e));
                else n4 = make_int4(__ldg(nb), r.deg > 1 ? __ldg(nb + 1) : 0, 0, 0);   // cap 1 or 2
                const int left = r.deg - e;
                unsigned any = __ldca(fb + (n4.x >> 5)) >> (n4.x & 31);
                if (left > 1) any |= __ldca(fb + (n4.y >> 5)) >> (n4.y & 31);
                if (left > 2) any |= __ldca(fb + (n4.z >> 5)) >> (n4.z & 31);
                if (left > 3) any |= __ldca(fb + (n4.w >> 5)) >> (n4.w & 31);
                hit = any & 1u;
            }
            unsigned more = __ballot_sync(kFull, !hit && r.deg > kBuLane);
            while (more) {
                const int l = __ffs(more) - 1;
                more &= more - 1;
                const int32_t* wn = pool + __shfl_sync(kFull, r.off, l);
                const int wd = __shfl_sync(kFull, r.deg, l);
                bool got = false;
                for (int e = kBuLane; e < wd && !got; e += 64) {
                    const int x = e + lane < wd ? __ldg(wn + e + lane) : -1;
                    const int y = e + 32 + lane < wd ? __ldg(wn + e + 32 + lane) : -1;
                    unsigned any = x >= 0 ? __ldca(fb + (x >> 5)) >> (x & 31) : 0u;
                    any |= y >= 0 ? __ldca(fb + (y >> 5)) >> (y & 31) : 0u;
                    got = __any_sync(kFull, any & 1u);
                    beat += 64;
                    if (beat >= kBuBeat) {
                        if (lane == 0) grid_progress(&a.ctl->bar);
                        beat = 0;
                    }
                }
                if (lane == l) hit = got;
            }
            if (hit) {
                dist[v] = level;
                found++;
                queued += ((unsigned long long)(unsigned)r.deg << 32) | 1ull;   // deg > 0
            }
            const unsigned b = __ballot_sync(kFull, hit);
            if (lane == k) fresh = b;
        }
        if (own) {
            nfb[word] = fresh;
            if (fresh) bm[word] = vis | fresh;
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) queued += __shfl_xor_sync(kFull, queued, o);
    if (lane == 0 && queued) atomicAdd(cout, queued);
    return found;
}

// The queue of a frontier held as a bitmap (bottom-up -> top-down).
__device__ __noinline__ void queue_from_bits() {
    WarpSmem& sm = warp_smem();
    const LevelSmem& lo = level_smem();
    const unsigned* fb = lo.a.fbits[lo.fcur & 1];
    const int nV = lo.a.nV;
    const unsigned gw = grid_warp(), nwarps = grid_warps();
    const int lane = threadIdx.x & 31;
    const unsigned units = ((unsigned)nV + kWChunk - 1) >> kChunkShiftWarp;
    const unsigned nwords = ((unsigned)nV + 31) / 32;
    int nlist = 0, none = 0;
    for (unsigned c = gw; c < units; c += nwarps) {
        const unsigned word = c * kWIpt + lane;
        const unsigned mine = lane < kWIpt && word < nwords ? __ldcg(fb + word) : 0u;
        int w[kWIpt];
        unsigned claim = 0;
#pragma unroll
        for (int k = 0; k < kWIpt; k++) {
            w[k] = (int)((c << kChunkShiftWarp) + 32 * k + lane);
            if (__shfl_sync(0xFFFFFFFFu, mine, k) >> lane & 1u) claim |= 1u << k;
        }
        warp_claims<false>(sm, nlist, w, claim, lo, none);
    }
    if (nlist > 0) warp_flush<false>(sm, nlist, lo, none);
}

// CTA 0 alone: levels of at most kSmallEdges frontier edges, frontier and
// edge offsets in shared memory.  A level is two chains of memory accesses:
// the neighbours, then (together) their claims and their records.  Leaves
// when the frontier is empty or larger (then written to the queue arrays), or
// max_levels are run; the state is left in ctl->s_*.
__device__ __noinline__ int small_levels() {
    SmallSmem& sm = small_smem();
    const LevelSmem& lo = level_smem();
    const BfsArgs& a = lo.a;
    int found = 0;
    const unsigned kFull = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;
    BfsCtl* ctl = a.ctl;
    int nq = (int)(lo.cin & 0xFFFFFFFFull);
    unsigned total = (unsigned)(lo.cin >> 32);
    int level = lo.level;
    int cur = 0;
    long long ev = __ldcg(&ctl->edges_visited), scanned = __ldcg(&ctl->scanned);
    int left = __ldcg(&ctl->left);
    const VRec* __restrict__ vtab = a.vtab;
    const int32_t* __restrict__ pool = a.pool;
    unsigned* const bm = a.bitmap;
    int32_t* const dist = a.dist;
    BfsOut* const out = a.out;
    const int nV = a.nV;
    for (int i = threadIdx.x; i < nq; i += blockDim.x) {
        const unsigned o = __ldcg(a.qoff[lo.cur] + i);
        sm.off[0][i] = o;
        sm.base[0][i] = __ldcg(a.qbase[lo.cur] + i) - (long long)o;
    }
    if (threadIdx.x == 0) sm.off[0][nq] = total;
    __syncthreads();
    while (true) {
        const int nx = cur ^ 1;
        unsigned long long acc = 0;   // next frontier so far (uniform)
        // a warp takes rows of 32 consecutive edges, four at most a round; a
        // thin frontier occupies few warps and the others only wait at the
        // barriers (issue slots, not memory, bound a level that all warps run)
        for (unsigned e0 = 0; e0 < total; e0 += blockDim.x * 4) {
            const unsigned rows = (total - e0 + 31) / 32;
            const int active = rows < (unsigned)nwarps ? (int)rows : nwarps;
            int w[4];
            VRec r[4];
            bool claim[4];
            unsigned long long mine = 0, incl = 0;
            if (warp < active) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const unsigned row = e0 + (k * nwarps + warp) * 32;
                    w[k] = -1;
                    claim[k] = false;
                    if (row < total) {   // uniform
                        int s0 = 0;      // last entry starting at or before the row
                        for (int n = nq; n > 1;) {
                            const int step = (n + 31) / 32;
                            const bool le = lane * step < n && sm.off[cur][s0 + lane * step] <= row;
                            const int j = __popc(__ballot_sync(kFull, le)) - 1;
                            s0 += j * step;
                            n = n - j * step < step ? n - j * step : step;
                        }
                        const bool in = s0 + lane < nq;
                        const unsigned sj = in ? sm.off[cur][s0 + lane] : 0xFFFFFFFFu;
                        const unsigned rel = sj - row;
                        const unsigned bits =
                            __reduce_or_sync(kFull, in && sj > row && rel < 32u ? 1u << rel : 0u);
                        const int owner = s0 + __popc(bits & (kFull >> (31 - lane)));
                        const unsigned e = row + lane;
                        if (e < total) w[k] = __ldg(pool + sm.base[cur][owner] + e);
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (w[k] >= 0) {
                        const unsigned bit = 1u << (w[k] & 31);
                        const unsigned old = atomicOr(bm + (w[k] >> 5), bit);
                        r[k] = vtab[w[k]];
                        claim[k] = !(old & bit);
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (!claim[k]) continue;
                    dist[w[k]] = level;
                    found++;
                    // the next level reads the list after two barriers
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(pool + r[k].off));
                    if (r[k].deg) mine += ((unsigned long long)(unsigned)r[k].deg << 32) | 1ull;
                    else claim[k] = false;
                }
                incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned long long x = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += x;
                }
                if (lane == 31) sm.wsum[warp] = incl;
            }
            __syncthreads();
            if (warp < active) {
                unsigned long long before = acc, all = acc;
                for (int i = 0; i < active; i++) {
                    const unsigned long long x = sm.wsum[i];
                    if (i < warp) before += x;
                    all += x;
                }
                unsigned long long at = before + incl - mine;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (!claim[k]) continue;
                    const int pos = (int)(at & 0xFFFFFFFFull);
                    const unsigned off = (unsigned)(at >> 32);
                    sm.off[nx][pos] = off;
                    sm.base[nx][pos] = r[k].off - (long long)off;
                    at += ((unsigned long long)(unsigned)r[k].deg << 32) | 1ull;
                }
                if (threadIdx.x == 0) {
                    sm.next = all;
                    // the end (a further round's first entry overwrites it)
                    sm.off[nx][all & 0xFFFFFFFFull] = (unsigned)(all >> 32);
                }
            }
            __syncthreads();   // the entries are complete; wsum is free
            acc = sm.next;
        }
        // the level is over
        scanned += total;
        if (threadIdx.x == 0) {
            if (level <= kTraceLevels) {
                out->t_end[level - 1] = global_ns();
                out->lvl_edges[level - 1] = total;
            }
            // (a store: only this CTA works, and a 5 us level feels an atomic)
            *(volatile unsigned*)&ctl->bar.beat = (unsigned)level;
        }
        cur = nx;
        nq = (int)(acc & 0xFFFFFFFFull);
        total = (unsigned)(acc >> 32);
        ev += total;
        const bool last = nq == 0 || level >= nV;
        level++;
        left--;
        if (last || left == 0 || total > (unsigned)kSmallEdges) {
            // leave: the frontier in the queue arrays of buffer 0
            const unsigned nchunks = (total + kWChunk - 1) >> kChunkShiftWarp;
            const bool mark = nchunks <= 4096;
            if (!last) {
                for (int i = threadIdx.x; i <= nq; i += blockDim.x) {
                    const unsigned o = sm.off[cur][i];
                    a.qoff[0][i] = o;
                    if (i < nq) a.qbase[0][i] = sm.base[cur][i] + (long long)o;
                }
                if (mark)
                    for (unsigned c = threadIdx.x; c < nchunks; c += blockDim.x) {
                        int l = 0, h = nq;
                        while (h - l > 1) {
                            const int mid = (l + h) >> 1;
                            if (sm.off[cur][mid] <= c << kChunkShiftWarp) l = mid; else h = mid;
                        }
                        a.chunk[0][c] = l;
                    }
            }
            if (threadIdx.x == 0) {
                ctl->s_cin = acc;
                ctl->s_level = level;
                ctl->s_marks = mark ? 0 : 1;
                ctl->s_scanned = scanned;
                ctl->s_edges = ev;
                ctl->s_left = left;
                ctl->s_done = last ? 1 : 0;
                // a large frontier may go bottom-up at once
                const long long mu = a.m_total - ev;
                ctl->s_mode = a.alpha > 0 && total > (unsigned)kSmallEdges &&
                              (long long)total * a.alpha > mu;
            }
            return found;
        }
    }
}

// Grid barrier; the sealed state is then copied to every CTA's shared memory.
// After a wait that gave up, lo.error is set and the CTA leaves.
template <typename Seal>
__device__ __forceinline__ void grid_sync(const BfsArgs& a, Seal seal) {
    LevelSmem& lo = level_smem();
    BfsCtl* ctl = a.ctl;
    __syncthreads();
    if (threadIdx.x == 0) {
        if (!grid_barrier(&ctl->bar, lo.gen, a.wait_polls, seal)) {
            *(volatile int*)&a.out->error = HN_ERR_TIMEOUT;
            lo.error = 1;
        }
        lo.cin = __ldcg(&ctl->cin);
        lo.level = __ldcg(&ctl->level);
        lo.mode = __ldcg(&ctl->mode);
        lo.cur = __ldcg(&ctl->cur);
        lo.fcur = __ldcg(&ctl->fcur);
        lo.marks = __ldcg(&ctl->marks);
        lo.done = __ldcg(&ctl->done) || __ldcg(&ctl->left) <= 0;
        lo.nqbase = a.qbase[lo.cur ^ 1];
        lo.nqoff = a.qoff[lo.cur ^ 1];
        lo.nchunk = a.chunk[lo.cur ^ 1];
    }
    __syncthreads();
}

// One BFS (or its next max_levels levels).  DO: levels may run bottom-up.
template <bool DO>
__global__ void __launch_bounds__(kRunThreads, 1) k_bfs_run(const __grid_constant__ BfsArgs a) {
    LevelSmem& lo = level_smem();
    BfsCtl* ctl = a.ctl;
    volatile BfsCtl* vc = a.ctl;   // read and written by the CTA that seals a level
    int found = 0;
    if (threadIdx.x == 0) {
        lo.a = a;
        lo.vtab = a.vtab;
        lo.dist = a.dist;
        lo.cout = &ctl->cout;
        lo.error = 0;
        lo.gen = *(volatile unsigned*)&ctl->bar.gen;   // it moves only after this CTA arrives
    }
    if (a.first) {
        const int nV = a.nV, src = a.src;
        const long long t0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
        const long long nt = (long long)gridDim.x * blockDim.x;
        const long long nwords = ((long long)nV + 31) / 32;
        if ((reinterpret_cast<uintptr_t>(a.dist) & 15) == 0) {
            const int4 inf4 = make_int4(kInf, kInf, kInf, kInf);
            const long long n4 = nV / 4;
            for (long long i = t0; i < n4; i += nt) {
                int4 x = inf4;
                if (src >> 2 == i) {
                    if ((src & 3) == 0) x.x = 0;
                    if ((src & 3) == 1) x.y = 0;
                    if ((src & 3) == 2) x.z = 0;
                    if ((src & 3) == 3) x.w = 0;
                }
                reinterpret_cast<int4*>(a.dist)[i] = x;
            }
            for (long long i = n4 * 4 + t0; i < nV; i += nt) a.dist[i] = i == src ? 0 : kInf;
        } else {
            for (long long i = t0; i < nV; i += nt) a.dist[i] = i == src ? 0 : kInf;
        }
        for (long long i = t0; i < nwords; i += nt)
            a.bitmap[i] = i == src / 32 ? 1u << (src & 31) : 0u;
        const VRec r = a.vtab[src];
        const unsigned d = (unsigned)r.deg;
        // chunk marks of a high-degree source are spread over the grid
        for (long long c = t0; c < ((long long)d + kWChunk - 1) / kWChunk; c += nt)
            a.chunk[0][c] = 0;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.qbase[0][0] = r.off;
            a.qoff[0][0] = 0;
            a.qoff[0][d > 0 ? 1 : 0] = d;
            ctl->cin = d > 0 ? (((unsigned long long)d << 32) | 1ull) : 0ull;
            ctl->cout = 0;
            ctl->level = 1;
            ctl->mode = 0;
            ctl->cur = 0;
            ctl->fcur = 0;
            ctl->marks = 0;
            ctl->done = 0;
            ctl->left = a.max_levels;
            ctl->visited = 1;
            ctl->scanned = 0;
            ctl->edges_visited = d;
            a.out->t_start = global_ns();
        }
    } else if (blockIdx.x == 0 && threadIdx.x == 0) {
        ctl->left = a.max_levels;
        ctl->done = 0;
    }
    auto nothing = [] {};
    grid_sync(a, nothing);
    while (!lo.error) {
        if (DO && lo.mode == 0 && lo.fcur >= 2) {
            queue_from_bits();
            grid_sync(a, [&] {
                const unsigned long long cn = atomicExch(&ctl->cout, 0ull);
                vc->cur = vc->cur ^ 1;
                a.qoff[vc->cur][cn & 0xFFFFFFFFull] = (unsigned)(cn >> 32);
                vc->fcur = 0;
            });
            if (lo.error) break;
        }
        const unsigned total = (unsigned)(lo.cin >> 32);
        const int level = lo.level, cur = lo.cur;
        const bool thin = total <= 32u * grid_warps();
        if (lo.mode == 0 && total <= (unsigned)kSmallEdges) {
            if (blockIdx.x == 0)
                found = small_levels();
        } else {
            // chunk marks that the previous (small or thin) level left to the grid
            if (lo.marks && !thin && !(DO && lo.mode == 1)) {
                const int nq = (int)(lo.cin & 0xFFFFFFFFull);
                const unsigned nchunks = (total + kWChunk - 1) >> kChunkShiftWarp;
                for (unsigned c = blockIdx.x * blockDim.x + threadIdx.x; c < nchunks;
                     c += gridDim.x * blockDim.x) {
                    int l = 0, h = nq;
                    while (h - l > 1) {
                        const int mid = (l + h) >> 1;
                        if (__ldcg(a.qoff[cur] + mid) <= c << kChunkShiftWarp) l = mid; else h = mid;
                    }
                    a.chunk[cur][c] = l;
                }
                grid_sync(a, [&] { vc->marks = 0; });
                if (lo.error) break;
            }
            if (DO && lo.mode == 1) {
                if (lo.fcur < 2) {   // the frontier is a queue: its bitmap first
                    frontier_bits();
                    grid_sync(a, [&] { vc->fcur = 2; });
                    if (lo.error) break;
                }
                found = bottom_up_level();
            } else if (thin) {
                found = thin_level();
            } else {
                found = top_down_level();
            }
        }
        // the visited count, before the level is sealed
        int f = found;
        found = 0;
        for (int o = 16; o; o >>= 1) f += __shfl_down_sync(0xFFFFFFFFu, f, o);
        if ((threadIdx.x & 31) == 0 && f)
            atomicAdd((unsigned long long*)&ctl->visited, (unsigned long long)f);
        const bool small = lo.mode == 0 && total <= (unsigned)kSmallEdges;
        const int mode = lo.mode, fcur = lo.fcur;
        const int nq = (int)(lo.cin & 0xFFFFFFFFull);
        grid_sync(a, [&] {
            if (small) {
                vc->cin = vc->s_cin;
                vc->level = vc->s_level;
                vc->mode = vc->s_mode;
                vc->cur = 0;
                vc->marks = vc->s_marks;
                vc->done = vc->s_done;
                vc->left = vc->s_left;
                vc->scanned = vc->s_scanned;
                vc->edges_visited = vc->s_edges;
            } else {
                const unsigned long long cn = atomicExch(&ctl->cout, 0ull);
                const unsigned nn = (unsigned)(cn & 0xFFFFFFFFull);
                const long long mf = (long long)(cn >> 32);
                vc->cin = cn;
                vc->scanned = vc->scanned + total;
                vc->edges_visited = vc->edges_visited + mf;
                vc->level = level + 1;
                vc->left = vc->left - 1;
                vc->done = !(nn > 0 && level < a.nV);
                vc->marks = mode == 0 && thin ? 1 : 0;
                if (level <= kTraceLevels) {
                    a.out->t_end[level - 1] = global_ns();
                    a.out->lvl_edges[level - 1] = total;
                }
                int next = mode;
                if (DO) {
                    // Beamer's switch: to bottom-up when the next frontier's
                    // edges exceed 1/alpha of the unexplored edges (alpha = 4
                    // by default: 287 us a source at scale 22, 309 at 14,
                    // 302 at 1), back to top-down when the frontier falls
                    // below nV/beta vertices (beta = 24) and is shrinking; a
                    // frontier that fits CTA 0 is always top-down
                    const long long mu = a.m_total - vc->edges_visited;
                    if (mode == 0) {
                        if (mf * a.alpha > mu) next = 1;
                    } else if ((long long)nn * a.beta < a.nV && nn < (unsigned)nq) {
                        next = 0;
                    }
                    if (mf <= kSmallEdges) next = 0;
                }
                vc->mode = next;
                if (mode == 0) {
                    vc->cur = cur ^ 1;
                    a.qoff[cur ^ 1][nn] = (unsigned)mf;
                    vc->fcur = 0;
                } else {
                    // bit 1: the frontier is the bitmap fbits[bit 0]
                    vc->fcur = 2 | ((fcur & 1) ^ 1);
                }
            }
        });
        if (lo.error) break;
        if (lo.done) break;
    }
    if (!lo.error && blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->level = lo.level;
        a.out->done = vc->done;
        a.out->visited = (long long)atomicAdd((unsigned long long*)&ctl->visited, 0ull);
        a.out->scanned = vc->scanned;
    }
}

// One BFS level.  TopDown (always, or while st->mode == 0 when DO): the
// frontier's edges in chunks.  BottomUp (DO and st->mode == 1): every
// unvisited vertex scans its sorted neighbours for one at distance level-1
// and stops at the first (Beamer, Asanovic & Patterson, "Direction-Optimizing
// Breadth-First Search", SC 2012).  Both produce the next frontier queue, so
// the direction may change at any level; distances are the same either way.
template <bool DO>
__global__ void __launch_bounds__(kBfsBlock, 9)
k_bfs_level(BfsState* st, cudaGraphConditionalHandle cond) {
    __shared__ BfsSmem sm;
    const int level = st->level;
    const int it = level - 1;
    const unsigned long long cin = st->cnt[it % 3];
    unsigned long long* cout = &st->cnt[(it + 1) % 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) st->cnt[(it + 2) % 3] = 0;
    const int nq = (int)(cin & 0xFFFFFFFFull);
    const unsigned total = (unsigned)(cin >> 32);
    const int cur = it & 1, nxt = cur ^ 1;
    int32_t* nqv = st->q[nxt];
    long long* nqbase = st->qbase[nxt];
    unsigned* nqoff = st->qoff[nxt];
    int32_t* nchunk = st->chunk[nxt];
    const VRec* vtab = st->vtab;
    const int32_t* pool = st->pool;
    unsigned* bm = st->bitmap;
    int32_t* dist = st->dist;
    const int mode = DO ? st->mode : 0;
    int found = 0;

    if (mode == 0) {
        const long long* qbase = st->qbase[cur];
        const unsigned* qoff = st->qoff[cur];
        const int32_t* chunk = st->chunk[cur];
        const unsigned nchunks = (total + kChunk - 1) / kChunk;
        const bool dyn = st->dynamic_chunks != 0;
        const bool warp_strided = st->warp_strided != 0;
        if (threadIdx.x == 0) sm.next = dyn ? atomicAdd(&st->next_chunk, 1u) : blockIdx.x;
        __syncthreads();
        for (unsigned c = sm.next; c < nchunks; c = sm.next) {
            const unsigned e0 = c * kChunk;
            const unsigned e1 = e0 + kChunk < total ? e0 + kChunk : total;
            const int s0 = chunk[c];
            const int s1 = c + 1 < nchunks ? chunk[c + 1] : nq - 1;   // inclusive
            const int nw = s1 - s0 + 1;
            for (int j = threadIdx.x; j <= nw; j += kBfsBlock) {
                int s = s0 + j;
                unsigned so = qoff[s];        // qoff[nq] is the sealed total
                sm.start[j] = so;
                if (j < nw) sm.base[j] = qbase[s] - (long long)so;
            }
            if (threadIdx.x == 0) sm.nw = nw;
            __syncthreads();
            int w[kIpt];
            bool claim[kIpt];
#pragma unroll
            for (int k = 0; k < kIpt; k++) { w[k] = -1; claim[k] = false; }
            bool mine_any = false;
            if (warp_strided) {
                // the warp's 32*kIpt edges, lane-strided: each load reads 32
                // consecutive edges (one window for high-degree vertices);
                // windows are searched inside the warp's own window range
                const unsigned wb = e0 + (threadIdx.x >> 5) * (32 * kIpt);
                if (wb < e1) {
                    const unsigned wl = wb + 32 * kIpt - 1 < e1 - 1 ? wb + 32 * kIpt - 1 : e1 - 1;
                    int jw0 = 0, jw1 = 0;
                    {
                        int lo = 0, hi = sm.nw;   // last j with start[j] <= wb
                        while (hi - lo > 1) {
                            int mid = (lo + hi) >> 1;
                            if (sm.start[mid] <= wb) lo = mid; else hi = mid;
                        }
                        jw0 = lo;
                        hi = sm.nw;               // last j with start[j] <= wl
                        while (hi - lo > 1) {
                            int mid = (lo + hi) >> 1;
                            if (sm.start[mid] <= wl) lo = mid; else hi = mid;
                        }
                        jw1 = lo;
                    }
#pragma unroll
                    for (int k = 0; k < kIpt; k++) {
                        const unsigned e = wb + k * 32 + (threadIdx.x & 31);
                        if (e < e1) {
                            int lo = jw0, hi = jw1 + 1;
                            while (hi - lo > 1) {
                                int mid = (lo + hi) >> 1;
                                if (sm.start[mid] <= e) lo = mid; else hi = mid;
                            }
                            w[k] = __ldg(pool + sm.base[lo] + e);
                            mine_any = true;
                        }
                    }
                }
            } else {
                // this thread's edges [a, b)
                const unsigned a = e0 + threadIdx.x * kIpt;
                const unsigned b = a + kIpt < e1 ? a + kIpt : e1;
                if (a < b) {
                    mine_any = true;
                    int lo = 0, hi = sm.nw;        // last j with start[j] <= a
                    while (hi - lo > 1) {
                        int mid = (lo + hi) >> 1;
                        if (sm.start[mid] <= a) lo = mid; else hi = mid;
                    }
                    int j = lo;
#pragma unroll
                    for (int k = 0; k < kIpt; k++) {
                        unsigned e = a + k;
                        if (e < b) {
                            while (sm.start[j + 1] <= e) j++;
                            w[k] = __ldg(pool + sm.base[j] + e);
                        }
                    }
                }
            }
            if (mine_any) {
                unsigned word[kIpt];
#pragma unroll
                for (int k = 0; k < kIpt; k++)
                    word[k] = w[k] >= 0 ? __ldca(bm + (w[k] >> 5)) : 0xFFFFFFFFu;
#pragma unroll
                for (int k = 0; k < kIpt; k++) {
                    if (w[k] >= 0 && !(word[k] & (1u << (w[k] & 31)))) {
                        unsigned bit = 1u << (w[k] & 31);
                        claim[k] = !(atomicOr(bm + (w[k] >> 5), bit) & bit);
                    }
                }
            }
            bfs_enqueue(sm, w, claim, level, vtab, dist, cout, nqv, nqbase, nqoff, nchunk,
                        kChunkShiftCta, found);
            // bfs_enqueue ends with a barrier, so every thread has read sm.next
            if (threadIdx.x == 0) sm.next = dyn ? atomicAdd(&st->next_chunk, 1u) : c + gridDim.x;
            __syncthreads();
        }
    } else {
        // bottom-up over all vertices, kIpt per thread, striped
        const int nV = st->nV;
        const int per = kBfsBlock * kIpt;
        const int nvc = (nV + per - 1) / per;
        for (int c = blockIdx.x; c < nvc; c += gridDim.x) {
            int w[kIpt];
            bool claim[kIpt];
            int dv[kIpt];
#pragma unroll
            for (int k = 0; k < kIpt; k++) {
                int v = c * per + k * kBfsBlock + threadIdx.x;
                w[k] = v < nV ? v : -1;
                claim[k] = false;
                dv[k] = w[k] >= 0 ? __ldcg(dist + v) : 0;
            }
#pragma unroll
            for (int k = 0; k < kIpt; k++) {
                if (w[k] >= 0 && dv[k] == kInf) {
                    VRec r = vtab[w[k]];
                    const int32_t* nb = pool + r.off;
                    for (int i = 0; i < r.deg; i++) {
                        if (__ldca(dist + nb[i]) == level - 1) { claim[k] = true; break; }
                    }
                    if (claim[k]) atomicOr(bm + (w[k] >> 5), 1u << (w[k] & 31));
                }
            }
            bfs_enqueue(sm, w, claim, level, vtab, dist, cout, nqv, nqbase, nqoff, nchunk,
                        kChunkShiftCta, found);
        }
    }
    bfs_level_end<DO>(st, cond, found, level, nq, total, cout, nqoff);
}

// The device arrays, and for bfs.kernel = 0 the CUDA graphs.
void build_bfs_graph(hn_graph* g, BfsGraph& bg) {
    const int nV = g->nV;
    // the finer of the two granularities, with room for the graph to grow
    // by a quarter before the arrays (and CUDA graphs) are rebuilt
    const long long nchunk_cap = (g->nE + g->nE / 4) / kWChunk + 1024;
    const size_t nwords = ((size_t)nV + 31) / 32 + 1;
    size_t bytes = 0;
    auto carve = [&](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) & ~(size_t)255;
        return at;
    };
    const size_t o_qbase = carve(sizeof(long long) * 2 * ((size_t)nV + 1));
    const size_t o_qoff = carve(sizeof(unsigned) * 2 * ((size_t)nV + 2));
    const size_t o_chunk = carve(sizeof(int32_t) * 2 * (size_t)nchunk_cap);
    const size_t o_bitmap = carve(sizeof(unsigned) * nwords);
    const size_t o_fbits = carve(bg.kernel ? sizeof(unsigned) * 2 * nwords : 0);
    const size_t o_ctl = carve(sizeof(BfsCtl));
    const size_t o_state = carve(sizeof(BfsState));
    const size_t o_q = carve(bg.kernel ? 0 : sizeof(int32_t) * 2 * ((size_t)nV + 1));
    HN_CUDA(cudaMallocAsync((void**)&bg.mem, bytes, g->stream));
    bg.qbasebuf = (long long*)(bg.mem + o_qbase);
    bg.qoffbuf = (unsigned*)(bg.mem + o_qoff);
    bg.chunkbuf = (int32_t*)(bg.mem + o_chunk);
    bg.bitmap = (unsigned*)(bg.mem + o_bitmap);
    bg.fbits = (unsigned*)(bg.mem + o_fbits);
    bg.ctl = (BfsCtl*)(bg.mem + o_ctl);
    bg.state = (BfsState*)(bg.mem + o_state);
    bg.qbuf = (int32_t*)(bg.mem + o_q);
    bg.nV = nV;
    bg.nchunk_cap = nchunk_cap;
    HN_CUDA(cudaMemsetAsync(bg.ctl, 0, sizeof(BfsCtl), g->stream));
    HN_CUDA(cudaMallocHost((void**)&bg.h_out, sizeof(BfsOut) * BfsGraph::kRing));
    HN_CUDA(cudaStreamCreateWithFlags(&bg.copy, cudaStreamNonBlocking));
    for (int b = 0; b < 2; b++) {
        HN_CUDA(cudaEventCreateWithFlags(&bg.done[b], cudaEventDisableTiming));
        HN_CUDA(cudaEventCreateWithFlags(&bg.copied[b], cudaEventDisableTiming));
    }
    if (bg.kernel) return;
    HN_CUDA(cudaMallocHost((void**)&bg.h_state, sizeof(BfsState)));
    HN_CUDA(cudaMallocHost((void**)&bg.h_ring, sizeof(BfsState) * BfsGraph::kRing));

    for (int variant = 0; variant < 2; variant++) {
        cudaGraph_t& graph = bg.graph[variant];
        HN_CUDA(cudaGraphCreate(&graph, 0));
        cudaGraphNode_t init_node, cond_node, body_node;
        {
            void* args[] = {&bg.state};
            cudaKernelNodeParams p = {};
            p.func = (void*)k_bfs3_init;
            p.gridDim = dim3((unsigned)grid_for(g, nV, 256));
            p.blockDim = dim3(256);
            p.kernelParams = args;
            HN_CUDA(cudaGraphAddKernelNode(&init_node, graph, nullptr, 0, &p));
        }
        cudaGraphConditionalHandle handle;
        HN_CUDA(cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault));
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = handle;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        HN_CUDA(cudaGraphAddNode(&cond_node, graph, &init_node, 1, &cp));
        cudaGraph_t body = cp.conditional.phGraph_out[0];
        {
            void* args[] = {&bg.state, &handle};
            cudaKernelNodeParams p = {};
            p.func = variant ? (void*)k_bfs_level<true> : (void*)k_bfs_level<false>;
            p.gridDim = dim3(bg.grid);
            p.blockDim = dim3(bg.threads);
            p.kernelParams = args;
            HN_CUDA(cudaGraphAddKernelNode(&body_node, body, nullptr, 0, &p));
        }
        HN_CUDA(cudaGraphInstantiate(&bg.exec[variant], graph, 0));
    }
}

}  // namespace

void free_bfs_graph(BfsGraph* bg) {
    if (!bg) return;
    for (int i = 0; i < 2; i++) {
        if (bg->exec[i]) cudaGraphExecDestroy(bg->exec[i]);
        if (bg->graph[i]) cudaGraphDestroy(bg->graph[i]);
    }
    if (bg->copy) cudaStreamSynchronize(bg->copy);
    for (int i = 0; i < 2; i++) {
        if (bg->done[i]) cudaEventDestroy(bg->done[i]);
        if (bg->copied[i]) cudaEventDestroy(bg->copied[i]);
    }
    if (bg->copy) cudaStreamDestroy(bg->copy);
    if (bg->h_out) cudaFreeHost(bg->h_out);
    if (bg->h_ring) cudaFreeHost(bg->h_ring);
    if (bg->h_state) cudaFreeHost(bg->h_state);
    // every BFS call has synchronised its stream, so no kernel uses the arrays
    if (bg->mem) cudaFreeAsync(bg->mem, 0);
    delete bg;
}

namespace {

BfsGraph& bfs_graph_of(hn_graph* g) {
    // rebuilt when the vertex count changes, the edge count outgrows the
    // chunk table or a knob changes the kernel or its grid
    const int kernel = (int)knob(kKnobBfsKernel);
    unsigned grid, threads;
    if (kernel) {
        // one cooperative CTA per SM, 256 threads for each of
        // bfs.warp_ctas_per_sm (three fill the registers)
        grid = (unsigned)g->info.sms;
        threads = 256u * (unsigned)std::min<long long>(knob(kKnobBfsWarpCtasPerSm), kRunThreads / 256);
    } else {
        grid = (unsigned)(g->info.sms * knob(kKnobBfsCtasPerSm));
        threads = kBfsBlock;
    }
    if (g->bfs && (g->bfs->nV != g->nV || g->nE / kWChunk + 4 > g->bfs->nchunk_cap ||
                   g->bfs->grid != grid || g->bfs->threads != threads ||
                   g->bfs->kernel != kernel)) {
        HN_CUDA(cudaStreamSynchronize(g->stream));
        free_bfs_graph(g->bfs);
        g->bfs = nullptr;
    }
    if (!g->bfs) {
        g->bfs = new BfsGraph();
        g->bfs->grid = grid;
        g->bfs->threads = threads;
        g->bfs->kernel = kernel;
        try {
            build_bfs_graph(g, *g->bfs);
        } catch (...) {
            free_bfs_graph(g->bfs);
            g->bfs = nullptr;
            throw;
        }
    }
    return *g->bfs;
}

constexpr int64_t kShareMax = 1 << 26;   // edges

hn_graph* bfs_root(hn_graph* g) { return g->parent ? g->parent : g; }

// Launches one BFS from `src` into `dist` with k_bfs_run; its result arrives
// in `out` (pinned).
void launch_run(hn_graph* g, BfsGraph& bg, int src, int32_t* dist, BfsOut* out,
                bool direction_optimizing) {
    cudaStream_t s = g->stream;
    // A cooperative launch of a CTA on every SM leaves no room for another one,
    // so BFS calls on several views would queue, though a small traversal has
    // work for few CTAs.  Each call takes its share of the SMs instead.  us per
    // BFS with 1 / 2 / 4 / 8 views at work, queued and shared: street grid 3390 /
    // 3370 / 3350 / 3350 and 3390 / 2120 / 1270 / 740; R-MAT scale 12 70 / 47 / 46
    // / 46 and 70 / 41 / 22 / 16, scale 16 91 / 72 / 71 / 78 and 93 / 50 / 28 / 20,
    // scale 20 234 / 214 / 214 / 216 and 232 / 177 / 155 / 141.  Larger ones fill
    // the GPU, and the second of two calls alone would have half of it (scale 22:
    // 278 queued, 259 / 220 / 195 shared; a request mix on scale 25 with 1,000
    // requests/s offered: 1,019 served queued, 944 shared).
    unsigned grid = bg.grid;
    if (g->nE <= kShareMax)
        grid = std::max(1u, grid / (unsigned)std::max(1, bfs_root(g)->bfs_running.load(
                                                             std::memory_order_relaxed)));
    void* fn = direction_optimizing ? (void*)k_bfs_run<true> : (void*)k_bfs_run<false>;
    // set per call: the attribute belongs to the device in use
    HN_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRunSmem));
    const size_t nwords = ((size_t)g->nV + 31) / 32 + 1;
    BfsArgs a;
    a.ctl = bg.ctl;
    a.out = out;
    a.vtab = g->vtab;
    a.pool = g->pool;
    a.dist = dist;
    a.bitmap = bg.bitmap;
    for (int b = 0; b < 2; b++) {
        a.fbits[b] = bg.fbits + b * nwords;
        a.qbase[b] = bg.qbasebuf + b * ((size_t)g->nV + 1);
        a.qoff[b] = bg.qoffbuf + b * ((size_t)g->nV + 2);
        a.chunk[b] = bg.chunkbuf + b * bg.nchunk_cap;
    }
    a.m_total = g->nE;
    a.nV = g->nV;
    a.src = src;
    a.alpha = direction_optimizing ? (int)knob(kKnobBfsDoAlpha) : 0;
    a.beta = (int)knob(kKnobBfsDoBeta);
    a.first = 1;
    *out = BfsOut{};
    // bfs.host_levels: one launch per level, so that each can be profiled
    const bool host_driven = knob(kKnobBfsHostLevels) != 0;
    a.max_levels = host_driven ? 1 : INT_MAX;
    a.wait_polls = (unsigned)knob(kKnobGridWaitPolls);
    cudaEvent_t ev0 = nullptr;
    if (g_profiling) profile_begin(s, &ev0);
    while (true) {
        void* args[] = {&a};
        HN_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(bg.threads), args, kRunSmem, s));
        count_launch();
        if (!host_driven) break;
        HN_CUDA(cudaStreamSynchronize(s));
        if (out->done || out->error) break;
        a.first = 0;
    }
    if (ev0) profile_end(direction_optimizing ? "k_bfs_run<true>" : "k_bfs_run<false>", s, ev0);
}

// The same with the CTA-chunk level kernel in its CUDA graph; the finished
// state arrives in `h` (pinned).
void launch_levels(hn_graph* g, BfsGraph& bg, int src, int32_t* dist, BfsState& h,
                   bool direction_optimizing) {
    cudaStream_t s = g->stream;
    const int nV = g->nV;
    const bool host_driven = knob(kKnobBfsHostLevels) != 0;
    h = BfsState{};
    h.src = src;
    h.nV = nV;
    h.dist = dist;
    h.vtab = g->vtab;
    h.pool = g->pool;
    h.q[0] = bg.qbuf;
    h.q[1] = bg.qbuf + nV + 1;
    h.qbase[0] = bg.qbasebuf;
    h.qbase[1] = bg.qbasebuf + nV + 1;
    h.qoff[0] = bg.qoffbuf;
    h.qoff[1] = bg.qoffbuf + nV + 2;
    h.chunk[0] = bg.chunkbuf;
    h.chunk[1] = bg.chunkbuf + bg.nchunk_cap;
    h.bitmap = bg.bitmap;
    h.m_total = g->nE;
    h.alpha = (int)knob(kKnobBfsDoAlpha);
    h.beta = (int)knob(kKnobBfsDoBeta);
    h.dynamic_chunks = (int)knob(kKnobBfsDynamicChunks);
    h.warp_strided = (int)knob(kKnobBfsWarpStrided);
    h.host_driven = host_driven ? 1 : 0;
    h.next_chunk = 0;
    h.cshift = kChunkShiftCta;
    HN_CUDA(cudaMemcpyAsync(bg.state, &h, sizeof(BfsState), cudaMemcpyHostToDevice, s));
    // profiling records the whole graph (one init + one expand per level)
    // under the name of its dominant kernel
    cudaEvent_t ev0 = nullptr;
    if (g_profiling) profile_begin(s, &ev0);
    if (host_driven) {
        // host-driven levels: one ordinary launch per level (each level can
        // be profiled on its own), one host round trip per level
        k_bfs3_init<<<(unsigned)grid_for(g, nV, 256), 256, 0, s>>>(bg.state);
        HN_CUDA(cudaGetLastError());
        count_launch();
        for (int lv = 0; lv <= nV; lv++) {
            cudaGraphConditionalHandle none = 0;
            void* args[] = {&bg.state, &none};
            HN_CUDA(cudaLaunchKernel(direction_optimizing ? (void*)k_bfs_level<true>
                                                          : (void*)k_bfs_level<false>,
                                     dim3(bg.grid), dim3(bg.threads), args, 0, s));
            count_launch();
            HN_CUDA(cudaMemcpyAsync(&bg.h_state->cont, &bg.state->cont, sizeof(int),
                                    cudaMemcpyDeviceToHost, s));
            HN_CUDA(cudaStreamSynchronize(s));
            if (!bg.h_state->cont) break;
        }
    } else {
        HN_CUDA(cudaGraphLaunch(bg.exec[direction_optimizing ? 1 : 0], s));
        count_launch(2);
    }
    if (ev0) profile_end(direction_optimizing ? "k_bfs_level<true>" : "k_bfs_level<false>", s, ev0);
    // the finished state back into this source's ring slot (ordered before
    // the next source's state upload on the same stream)
    HN_CUDA(cudaMemcpyAsync(&h, bg.state, sizeof(BfsState), cudaMemcpyDeviceToHost, s));
}

void bfs_run(hn_graph* g, const int32_t* sources, int k, int32_t* dist, int mem,
             hn_bfs_stats_t* stats, bool direction_optimizing) {
    cudaStream_t s = g->stream;
    const int nV = g->nV;
    for (int i = 0; i < k; i++)
        if (sources[i] < 0 || sources[i] >= nV)
            throw Error(HN_ERR_INVALID, "BFS source outside [0, nV)");
    // edge offsets are 32-bit, and a chunk's end (offset + 256) must not wrap
    if (g->nE > 0xFFFFFE00ll) throw Error(HN_ERR_CAPACITY, "BFS needs nE < 2^32 - 512");
    if (k == 0) return;
    struct Running {
        std::atomic<int>& n;
        explicit Running(std::atomic<int>& c) : n(c) { n.fetch_add(1, std::memory_order_relaxed); }
        ~Running() { n.fetch_sub(1, std::memory_order_relaxed); }
    } running(bfs_root(g)->bfs_running);
    BfsGraph& bg = bfs_graph_of(g);
    const bool host_out = mem == HN_MEM_HOST;
    // host output: two device buffers; BFS i writes buffer i % 2 while the
    // copy stream drains buffer (i - 1) % 2 to the host
    DevBuf<int32_t> d_dist;
    if (host_out) d_dist.alloc((size_t)2 * nV, s);
    // an early end waits for the copies before d_dist and the caller's array go
    struct CopiesEnd {
        cudaStream_t copy;
        ~CopiesEnd() {
            if (copy) cudaStreamSynchronize(copy);
        }
    } copies_end{host_out ? bg.copy : nullptr};
    std::vector<BfsOut> res((size_t)k);
    // results of the ring entries of sources [from, to)
    auto collect = [&](int from, int to) {
        HN_CUDA(cudaStreamSynchronize(s));
        for (int i = from; i < to; i++) {
            const int r = i % BfsGraph::kRing;
            if (bg.kernel) {
                res[i] = bg.h_out[r];
                if (res[i].error) {
                    // the sources queued behind this one were refused at
                    // their first barrier (kGridDead), and have finished
                    HN_CUDA(cudaMemsetAsync(bg.ctl, 0, sizeof(BfsCtl), s));
                    HN_CUDA(cudaStreamSynchronize(s));
                    throw Error(HN_ERR_TIMEOUT, "BFS: a bounded wait gave up");
                }
            } else {
                const BfsState& h = bg.h_ring[r];
                BfsOut& o = res[i];
                o = BfsOut{};
                o.level = h.level;
                o.visited = h.visited;
                o.scanned = h.scanned;
                o.t_start = h.t_start;
                std::copy(h.t_end, h.t_end + kTraceLevels, o.t_end);
                std::copy(h.lvl_edges, h.lvl_edges + kTraceLevels, o.lvl_edges);
            }
        }
    };
    if (!bg.kernel) HN_CUDA(cudaStreamSynchronize(s));   // the ring's previous contents are read
    int first = 0;   // sources before it are collected
    for (int i = 0; i < k; i++) {
        const int r = i % BfsGraph::kRing;
        if (i > 0 && r == 0) {
            collect(first, i);
            first = i;
        }
        const int b = i & 1;
        int32_t* out = host_out ? d_dist.get() + (size_t)b * nV : dist + (size_t)i * nV;
        if (host_out && i >= 2) HN_CUDA(cudaStreamWaitEvent(s, bg.copied[b], 0));
        if (bg.kernel)
            launch_run(g, bg, sources[i], out, &bg.h_out[r], direction_optimizing);
        else
            launch_levels(g, bg, sources[i], out, bg.h_ring[r], direction_optimizing);
        if (host_out) {
            HN_CUDA(cudaEventRecord(bg.done[b], s));
            HN_CUDA(cudaStreamWaitEvent(bg.copy, bg.done[b], 0));
            HN_CUDA(cudaMemcpyAsync(dist + (size_t)i * nV, out, sizeof(int32_t) * nV,
                                    cudaMemcpyDeviceToHost, bg.copy));
            HN_CUDA(cudaEventRecord(bg.copied[b], bg.copy));
        }
    }
    if (host_out) HN_CUDA(cudaStreamSynchronize(bg.copy));
    collect(first, k);
    bg.last = res[k - 1];
    bg.have_last = true;
    if (stats)
        for (int i = 0; i < k; i++) {
            stats[i].levels = res[i].level - 1;
            stats[i].pad = 0;
            stats[i].visited = res[i].visited;
            stats[i].edges_scanned = res[i].scanned;
        }
}

}  // namespace
}  // namespace hn

using namespace hn;

extern "C" {

int hn_bfs(hn_graph_t* g, int32_t src, int32_t* dist, int mem, hn_bfs_stats_t* stats) {
    HN_API_BEGIN
    HN_REQUIRE(g && dist, "null argument");
    HN_REQUIRE(mem == HN_MEM_HOST || mem == HN_MEM_DEVICE, "bad memory kind");
    HN_REQUIRE(g->nV > 0, "empty graph");
    HandleUse use(g);
    HN_CUDA(cudaSetDevice(g->device));
    bfs_run(g, &src, 1, dist, mem, stats, false);
    HN_API_END
}

int hn_bfs_multi(hn_graph_t* g, const int32_t* sources, int32_t k, int32_t* dist, int mem,
                 hn_bfs_stats_t* stats) {
    HN_API_BEGIN
    HN_REQUIRE(g && sources && dist, "null argument");
    HN_REQUIRE(k >= 0, "negative source count");
    HN_REQUIRE(mem == HN_MEM_HOST || mem == HN_MEM_DEVICE, "bad memory kind");
    HN_REQUIRE(g->nV > 0 || k == 0, "empty graph");
    HandleUse use(g);
    HN_CUDA(cudaSetDevice(g->device));
    bfs_run(g, sources, k, dist, mem, stats, false);
    HN_API_END
}

int hn_bfs_level_trace(hn_graph_t* g, int32_t max_levels, double* us, int64_t* edges,
                       int32_t* n_levels) {
    HN_API_BEGIN
    HN_REQUIRE(g && n_levels && max_levels >= 0, "null argument");
    *n_levels = 0;
    if (!g->bfs || !g->bfs->have_last) return HN_OK;
    const BfsOut& t = g->bfs->last;
    const int lv = t.level - 1 < kTraceLevels ? t.level - 1 : kTraceLevels;
    const int n = lv < max_levels ? lv : max_levels;
    unsigned long long prev = t.t_start;
    for (int i = 0; i < n; i++) {
        if (us) us[i] = (double)(t.t_end[i] - prev) / 1e3;
        if (edges) edges[i] = (int64_t)t.lvl_edges[i];
        prev = t.t_end[i];
    }
    *n_levels = n;
    HN_API_END
}

int hn_bfs_do(hn_graph_t* g, const int32_t* sources, int32_t k, int32_t* dist, int mem,
              hn_bfs_stats_t* stats) {
    HN_API_BEGIN
    HN_REQUIRE(g && sources && dist, "null argument");
    HN_REQUIRE(k >= 0, "negative source count");
    HN_REQUIRE(mem == HN_MEM_HOST || mem == HN_MEM_DEVICE, "bad memory kind");
    HN_REQUIRE(g->nV > 0 || k == 0, "empty graph");
    HandleUse use(g);
    HN_CUDA(cudaSetDevice(g->device));
    bfs_run(g, sources, k, dist, mem, stats, true);
    HN_API_END
}

}  // extern "C"
