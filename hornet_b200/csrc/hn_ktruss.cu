// k-truss (hornetsnest/src/Static/KTruss/KTruss.cu:90-174,
// KTrussSupport.cu:375-468, KTrussOperators.cuh:16-38).
//
// Reference semantics: max_K starts at 3; findTrussOfK repeatedly
// recomputes every edge's support (triangles through it) from scratch and
// deletes all edges with support < max_K - 2 through a BatchUpdate erase,
// until a pass deletes nothing; if no edge is left max_K-- and stop,
// otherwise max_K++ on the peeled graph.  (The reference k-truss does not
// compile against the current core; the definition is what is kept.)
//
// Here the supports are computed once and then maintained incrementally:
// a round deletes the current frontier F (edges with support < K-2) and,
// for every triangle (e, e1, e2) of a frontier edge e whose other two edges
// are still alive, decrements the supports it destroys exactly once — if
// neither e1 nor e2 is in F both lose one; if exactly one of them is in F
// the remaining edge loses one, charged to the smaller of the two frontier
// edges; if both are in F nothing remains to update.  An edge whose support
// crosses from K-2 to K-3 joins the next frontier.  After the rounds the
// supports equal the from-scratch supports of the peeled graph, so the
// surviving edge sets, truss numbers and max_K are those of the reference
// loop.  Edge ids are positions in the sorted CSR; undirected edge state
// lives on the (u < v) position.
#include <optional>

#include <algorithm>
#include <climits>
#include <cstring>

#include "hn_graph.cuh"
#include "hn_gridsync.cuh"
#include "hn_tc.cuh"

namespace hn {
namespace {

constexpr int kB = 256;

// Device state of the host-driven peel rounds (ktruss.device_rounds = 0):
// every kernel of a round reads its arrays and counts from here.
struct KtPeel {
    const long long* off;     // current adjacency lists (rebuilt as edges die)
    const int32_t* adj;
    const int32_t* canon;
    int32_t* F;               // this round's frontier (canonical edge ids)
    int32_t* NF;              // the next round's frontier
    int nf;                   // |F|
    int nNF;                  // |NF| (appended atomically)
    int nheavy;               // frontier edges left to the heavy kernel
    int K;
    long long remaining;      // alive edges
    long long rounds;         // peel rounds run
};

// canonical (u < v) position of every directed edge; checks simplicity and
// symmetry.
__global__ void k_kt_canon(const long long* __restrict__ off, const int32_t* __restrict__ adj,
                           const int32_t* __restrict__ src, long long m,
                           int32_t* __restrict__ canon, int* __restrict__ err) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m;
         e += (long long)gridDim.x * blockDim.x) {
        int u = src[e], v = adj[e];
        bool bad = (u == v) || (e > off[u] && adj[e - 1] == v);
        long long c = e;
        if (u > v) {
            long long p = off[v] + lower_bound_dev(adj + off[v], off[v + 1] - off[v], u);
            if (p >= off[v + 1] || adj[p] != u) bad = true;
            c = p;
        }
        canon[e] = (int)c;
        if (bad) atomicExch(err, 1);
    }
}

// Canonical edges (u < v) start alive (their supports come from the
// triangle enumeration: every triangle, found once, credits its three edges).
__global__ void k_kt_init(const int32_t* __restrict__ adj, const int32_t* __restrict__ src,
                          long long m, unsigned char* __restrict__ alive,
                          int* __restrict__ nalive) {
    int mine = 0;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m;
         e += (long long)gridDim.x * blockDim.x) {
        const bool canon = src[e] < adj[e];
        alive[e] = canon ? 1 : 0;
        mine += canon ? 1 : 0;
    }
    for (int o = 16; o; o >>= 1) mine += __shfl_down_sync(0xFFFFFFFFu, mine, o);
    if ((threadIdx.x & 31) == 0 && mine) atomicAdd(nalive, mine);
}

// Positions of the current lists whose (canonical) edge is still alive.
// (alive as bytes, or state: alive iff INT_MAX)
__global__ void k_kt_live_pos(const int32_t* __restrict__ canon, long long n,
                              const unsigned char* __restrict__ alive,
                              const int32_t* __restrict__ state, int32_t* __restrict__ flag) {
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < n;
         p += (long long)gridDim.x * blockDim.x)
        flag[p] = state ? state[canon[p]] == INT_MAX : alive[canon[p]] != 0;
}

// List shrinking: a vertex's new offset is the new slot of its first old
// entry (noff[v] = pos[off[v]], v = 0..nV), and every live entry moves to
// its new slot, in order.
__global__ void k_kt_shrink_off(const long long* __restrict__ off, int nV,
                                const long long* __restrict__ pos, long long* __restrict__ noff) {
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v <= nV;
         v += (long long)gridDim.x * blockDim.x)
        noff[v] = pos[off[v]];
}

__global__ void k_kt_shrink_copy(const int32_t* __restrict__ adj, const int32_t* __restrict__ canon,
                                 const int32_t* __restrict__ flag, const long long* __restrict__ pos,
                                 long long m, int32_t* __restrict__ nadj,
                                 int32_t* __restrict__ ncanon) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < m;
         i += (long long)gridDim.x * blockDim.x)
        if (flag[i]) {
            nadj[pos[i]] = adj[i];
            ncanon[pos[i]] = canon[i];
        }
}

// Frontier of round K: alive edges of the list L with support < K - 2.
__global__ void k_kt_frontier(const int32_t* __restrict__ L, int nL,
                              const int32_t* __restrict__ sup,
                              const unsigned char* __restrict__ alive,
                              unsigned char* __restrict__ inF, KtPeel* st) {
    const int K = st->K;
    int32_t* F = st->F;
    int* nF = &st->nf;
    for (long long i0 = blockIdx.x * (long long)blockDim.x; i0 < nL;
         i0 += (long long)gridDim.x * blockDim.x) {
        long long i = i0 + threadIdx.x;
        int e = i < nL ? L[i] : 0;
        bool take = i < nL && alive[e] && sup[e] < K - 2;
        int p = warp_append(nF, take);
        if (take) {
            F[p] = e;
            inF[e] = 1;
        }
    }
}

// Alive-edge list: from all canonical edges (L == nullptr, n = m) or from
// the previous list, dropping peeled edges; *minsup receives the smallest
// support left, so the next round can start at the first K that peels.
__global__ void k_kt_compact(const int32_t* __restrict__ L, long long n,
                             const unsigned char* __restrict__ alive,
                             const int32_t* __restrict__ sup, int32_t* __restrict__ out,
                             int* __restrict__ nout, int* __restrict__ minsup) {
    int mn = 0x7FFFFFFF;
    for (long long i0 = blockIdx.x * (long long)blockDim.x; i0 < n;
         i0 += (long long)gridDim.x * blockDim.x) {
        long long i = i0 + threadIdx.x;
        int e = i < n ? (L ? L[i] : (int)i) : 0;
        bool take = i < n && alive[e];
        int p = warp_append(nout, take);
        if (take) {
            out[p] = e;
            mn = min(mn, sup[e]);
        }
    }
    for (int o = 16; o; o >>= 1) mn = min(mn, __shfl_down_sync(0xFFFFFFFFu, mn, o));
    if ((threadIdx.x & 31) == 0 && mn != 0x7FFFFFFF) atomicMin(minsup, mn);
}

__device__ __forceinline__ void kt_dec(int x, int K, int32_t* sup, int32_t* NF, int* nNF) {
    int old = atomicSub(sup + x, 1);
    if (old == K - 2) NF[atomicAdd(nNF, 1)] = x;
}

// One common neighbour w of a frontier edge e = (u, v): e1 = (u, w) or
// (v, w) and e2 the other, in canonical ids.  Each destroyed triangle is
// charged exactly once (see the decrement rule above).
__device__ __forceinline__ void kt_triangle(int e, int e1, int e2, int K,
                                            const unsigned char* __restrict__ alive,
                                            const unsigned char* __restrict__ inF,
                                            int32_t* sup, int32_t* NF, int* nNF) {
    if (!alive[e1] || !alive[e2]) return;
    bool f1 = inF[e1], f2 = inF[e2];
    if (!f1 && !f2) {
        kt_dec(e1, K, sup, NF, nNF);
        kt_dec(e2, K, sup, NF, nNF);
    } else if (f1 && !f2) {
        if (e < e1) kt_dec(e2, K, sup, NF, nNF);
    } else if (!f1 && f2) {
        if (e < e2) kt_dec(e1, K, sup, NF, nNF);
    }
}

// Frontier edges whose shorter list has at most 32 entries: a thread each.
// Longer ones go to a list for k_kt_peel_heavy (a CTA each): the dense
// core's hub-hub edges would otherwise run one long intersection per thread.
__global__ void k_kt_peel(KtPeel* st, const int32_t* __restrict__ src,
                          const int32_t* __restrict__ eadj,
                          const unsigned char* __restrict__ alive,
                          const unsigned char* __restrict__ inF, int32_t* __restrict__ sup,
                          int32_t* __restrict__ heavy) {
    const long long* __restrict__ off = st->off;
    const int32_t* __restrict__ adj = st->adj;
    const int32_t* __restrict__ canon = st->canon;
    const int32_t* __restrict__ F = st->F;
    const int nF = st->nf, K = st->K;
    int32_t* NF = st->NF;
    int* nNF = &st->nNF;
    int* nheavy = &st->nheavy;
    for (long long f0 = blockIdx.x * (long long)blockDim.x; f0 < nF;
         f0 += (long long)gridDim.x * blockDim.x) {
        const long long f = f0 + threadIdx.x;
        bool big = false;
        int e = 0;
        if (f < nF) {
            e = F[f];
            int u = src[e], v = eadj[e];
            long long au = off[u], la = off[u + 1] - au;
            long long bv = off[v], lb = off[v + 1] - bv;
            bool swapped = la > lb;
            long long pa = swapped ? bv : au, pb = swapped ? au : bv;
            long long na = swapped ? lb : la, nb = swapped ? la : lb;
            if (na > 32) {
                big = true;
            } else {
                long long lo = 0;
                for (long long i = 0; i < na && lo < nb; i++) {
                    int w = adj[pa + i];
                    long long p = lo + lower_bound_dev(adj + pb + lo, nb - lo, w);
                    lo = p;
                    if (p >= nb || adj[pb + p] != w) continue;
                    lo = p + 1;
                    kt_triangle(e, canon[pa + i], canon[pb + p], K, alive, inF, sup, NF, nNF);
                }
            }
        }
        int slot = warp_append(nheavy, big);
        if (big) heavy[slot] = e;
    }
}

__global__ void k_kt_peel_heavy(KtPeel* st, const int32_t* __restrict__ src,
                                const int32_t* __restrict__ eadj,
                                const int32_t* __restrict__ heavy,
                                const unsigned char* __restrict__ alive,
                                const unsigned char* __restrict__ inF, int32_t* __restrict__ sup) {
    const long long* __restrict__ off = st->off;
    const int32_t* __restrict__ adj = st->adj;
    const int32_t* __restrict__ canon = st->canon;
    const int K = st->K;
    int32_t* NF = st->NF;
    int* nNF = &st->nNF;
    // a CTA per heavy edge: its shorter list is searched by all threads,
    // so a round whose frontier is a few hub-hub edges still spreads them
    const long long nh = st->nheavy;
    for (long long h = blockIdx.x; h < nh; h += gridDim.x) {
        const int e = heavy[h];
        const int u = src[e], v = eadj[e];
        const long long au = off[u], la = off[u + 1] - au;
        const long long bv = off[v], lb = off[v + 1] - bv;
        const bool swapped = la > lb;
        const long long pa = swapped ? bv : au, pb = swapped ? au : bv;
        const long long na = swapped ? lb : la, nb = swapped ? la : lb;
        for (long long i = threadIdx.x; i < na; i += blockDim.x) {
            const int w = adj[pa + i];
            const long long p = lower_bound_dev(adj + pb, nb, w);
            if (p < nb && adj[pb + p] == w)
                kt_triangle(e, canon[pa + i], canon[pb + p], K, alive, inF, sup, NF, nNF);
        }
    }
}

__global__ void k_kt_retire(const KtPeel* st, unsigned char* __restrict__ alive,
                            unsigned char* __restrict__ inF, int32_t* __restrict__ truss) {
    const int32_t* __restrict__ F = st->F;
    const int nF = st->nf, K = st->K;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nF;
         i += (long long)gridDim.x * blockDim.x) {
        int e = F[i];
        alive[e] = 0;
        inF[e] = 0;
        truss[e] = K - 1;
    }
}

__global__ void k_kt_mark(const KtPeel* st, unsigned char* __restrict__ inF) {
    const int32_t* __restrict__ NF = st->NF;
    const int nn = st->nNF;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nn;
         i += (long long)gridDim.x * blockDim.x)
        inF[NF[i]] = 1;
}

// End of a round (one thread): the peeled edges leave the alive count and the
// next frontier becomes the current one.
__global__ void k_kt_advance(KtPeel* st) {
    st->remaining -= st->nf;
    st->rounds++;
    int32_t* t = st->F;
    st->F = st->NF;
    st->NF = t;
    st->nf = st->nNF;
    st->nNF = 0;
    st->nheavy = 0;
}

// Start of a K (one thread): its value, empty frontier counters.
__global__ void k_kt_begin(KtPeel* st, int K) {
    st->K = K;
    st->nf = 0;
    st->nNF = 0;
    st->nheavy = 0;
}

// ---------------------------------------------------------------------------
// k_kt_run: the peel rounds of K after K in one cooperative launch
// (ktruss.device_rounds = 1).  A K ends with the compaction of the alive
// list, which also gives the next K that peels anything.  The kernel returns
// when no edge is left or when at most half of the entries of the adjacency
// lists are alive (the host then rebuilds the lists).
//
// Most rounds are small (a hundred thousand vertices: 62 values of K, several
// hundred rounds of a few edges), so what counts is the length of a round's
// chain of dependent steps:
//   * one grid barrier a round.  There is no retire or mark pass: state[e] is
//     kAlive or the round in which e is (or was) on the frontier, so in round
//     r an edge is on the frontier iff state = r, dead iff state < r, and an
//     edge that drops below K - 2 now gets state r + 1 and its truss number
//     when it is appended.  Frontiers and their sizes are indexed by the
//     round, so ending one takes no copying: the barrier's last CTA clears
//     one counter;
//   * a frontier of at most kKtFew edges is staged by every CTA for itself
//     (endpoints and list bounds, with the prefix of their 32-entry chunks),
//     and the chunks go round-robin to all warps, one binary search a lane;
//   * a frontier of at most kKtSolo edges is peeled by CTA 0 alone, and so are
//     the ones it leads to until one exceeds kKtSoloMax, without a grid
//     barrier.  CTA 0 leaves the shared state alone meanwhile (others may
//     still be reading it): the barrier's seal takes its result over;
//   * a larger frontier is split evenly over the CTAs, each staging its edges
//     (at most kKtFew at a time) and spreading their chunks over its warps.
// 100,003 vertices, 2.2 M edges, 62 values of K, 663 rounds: 29.7 ms with a
// WHILE node around five kernels a round, 13.3 ms with one barrier a round and
// a warp per large frontier's edge, 9.2 ms this way.
// ---------------------------------------------------------------------------
constexpr int kKtThreads = 1024;
constexpr int kKtFew = 512;      // edges staged per CTA
constexpr int kKtSolo = 16;      // edges that CTA 0 takes alone
constexpr int kKtSoloMax = 64;
constexpr int kKtBeat = 512;     // chunks of a warp between two signs of progress (2 ms with lists of 4 M)
static_assert(kKtSoloMax <= kKtFew, "CTA 0 stages its frontiers");
constexpr int kAlive = INT_MAX;

struct KtCtl {
    GridBar bar;
    // read by every CTA after a barrier
    int round;                // number of the current round, from 1
    int nL;                   // alive edges at the start of this K
    int K;
    int stop;
    int cnt[3];               // |frontier of round r| at [r % 3]
    int side;                 // the list L is L[side]
    int nL2, minsup, error;
    int x_round, x_nf;        // CTA 0's round and frontier after its rounds alone
};

struct KtArgs {
    KtCtl* ctl;
    const long long* off;     // adjacency lists (dead entries stay until rebuilt)
    const int32_t* adj;
    const int32_t* canon;
    long long lm;             // entries of adj
    int32_t* F[2];            // frontier of round r (canonical edge ids) at [r % 2]
    int32_t* L[2];            // alive edges of this K, and of the next
    const int32_t* src;       // endpoints of each edge id
    const int32_t* eadj;
    int32_t* state;
    int32_t* sup;
    int32_t* truss;
    unsigned wait_polls;      // limit of a wait at the grid barrier
};

// x loses a triangle; the thread that takes it below K - 2 puts it on the
// next frontier.
__device__ __forceinline__ void kt_drop(const KtArgs& a, int x, int K, int round, int* n_next) {
    if (atomicSub(a.sup + x, 1) == K - 2) {
        a.state[x] = round + 1;
        a.truss[x] = K - 1;
        a.F[(round + 1) & 1][atomicAdd(n_next, 1)] = x;
    }
}

// kt_triangle for the states above (read through L2: they change during the
// launch).
__device__ __forceinline__ void kt_common(const KtArgs& a, int e, int e1, int e2, int K, int round,
                                          int* n_next) {
    const int s1 = __ldcg(a.state + e1), s2 = __ldcg(a.state + e2);
    if (s1 < round || s2 < round) return;   // the triangle is already gone
    const bool f1 = s1 == round, f2 = s2 == round;
    if (!f1 && !f2) {
        kt_drop(a, e1, K, round, n_next);
        kt_drop(a, e2, K, round, n_next);
    } else if (f1 && !f2) {
        if (e < e1) kt_drop(a, e2, K, round, n_next);
    } else if (!f1 && f2) {
        if (e < e2) kt_drop(a, e1, K, round, n_next);
    }
}

__device__ __forceinline__ int kt_lower(const int32_t* __restrict__ a, int n, int x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(a + mid) < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

struct KtEdge {   // a frontier edge: the shorter list [pa, pa + na), the longer one
    int e, pa, pb, na, nb;
};

__device__ __forceinline__ KtEdge kt_edge(const KtArgs& a, const long long* __restrict__ off, int e) {
    KtEdge k;
    const int u = __ldg(a.src + e), v = __ldg(a.eadj + e);
    const int au = (int)__ldg(off + u), la = (int)__ldg(off + u + 1) - au;
    const int bv = (int)__ldg(off + v), lb = (int)__ldg(off + v + 1) - bv;
    const bool sw = la > lb;
    k.e = e;
    k.pa = sw ? bv : au;
    k.pb = sw ? au : bv;
    k.na = sw ? lb : la;
    k.nb = sw ? la : lb;
    return k;
}

__global__ void __launch_bounds__(kKtThreads, 1) k_kt_run(const __grid_constant__ KtArgs a) {
    __shared__ int s_nf, s_round, s_nL, s_K, s_stop, s_side, s_error, s_next;
    __shared__ unsigned s_gen;
    __shared__ int s_e[kKtFew], s_pa[kKtFew], s_pb[kKtFew], s_na[kKtFew], s_nb[kKtFew];
    __shared__ int s_pre[kKtFew + 1], s_ws[kKtFew / 32];
    const unsigned kFull = 0xFFFFFFFFu;
    KtCtl* ctl = a.ctl;
    volatile KtCtl* vc = a.ctl;   // read and written by the CTA that seals a phase
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int NW = kKtThreads / 32;
    const int gw = blockIdx.x * NW + warp;
    const int nwarps = gridDim.x * NW;
    const long long gt = blockIdx.x * (long long)kKtThreads + threadIdx.x;
    const long long nt = (long long)gridDim.x * kKtThreads;
    const int32_t* __restrict__ adj = a.adj;
    const int32_t* __restrict__ canon = a.canon;
    // after a barrier: the sizes that this round needs
    auto load = [&] {
        const int r = __ldcg(&ctl->round);
        s_nL = __ldcg(&ctl->nL);
        s_K = __ldcg(&ctl->K);
        s_stop = __ldcg(&ctl->stop);
        s_side = __ldcg(&ctl->side);
        s_nf = __ldcg(&ctl->cnt[r % 3]);
        s_round = r;
    };
    auto sync = [&](auto seal) {
        __syncthreads();
        if (threadIdx.x == 0) {
            if (!grid_barrier(&ctl->bar, s_gen, a.wait_polls, seal)) {
                *(volatile int*)&ctl->error = HN_ERR_TIMEOUT;
                s_error = 1;
            }
            load();
        }
        __syncthreads();
        return s_error == 0;
    };
    auto nothing = [] {};
    if (threadIdx.x == 0) {
        s_error = 0;
        s_gen = *(volatile unsigned*)&ctl->bar.gen;   // it moves only after this CTA arrives
        load();
    }
    __syncthreads();
    int beat = 0;   // chunks since this warp's last sign of progress
    while (true) {
        // the frontier of K: alive edges with support < K - 2
        {
            const int nL = s_nL, K = s_K, round = s_round;
            const int32_t* L = a.L[s_side];
            int* nf = &ctl->cnt[round % 3];
            for (long long i0 = gt - lane; i0 < nL; i0 += nt) {
                const long long i = i0 + lane;
                const int e = i < nL ? __ldcg(L + i) : 0;
                const bool take = i < nL && __ldcg(a.sup + e) < K - 2;
                const int p = warp_append(nf, take);
                if (take) {
                    a.F[round & 1][p] = e;
                    a.state[e] = round;
                    a.truss[e] = K - 1;
                }
            }
            if (!sync(nothing)) return;
        }
        while (s_nf > 0) {
            const int nf = s_nf, K = s_K, round = s_round;
            // entry i of the shorter list of frontier edge e of round r
            auto probe = [&](int e, int pa, int pb, int nb, int i, int r, int* n_next) {
                const int w = __ldg(adj + pa + i);
                const int p = kt_lower(adj + pb, nb, w);
                if (p < nb && __ldg(adj + pb + p) == w)
                    kt_common(a, e, __ldg(canon + pa + i), __ldg(canon + pb + p), K, r, n_next);
            };
            // round r for n <= kKtFew edges of its frontier, from f0 on, by the
            // warps first, first + step, ... (called by the whole CTA)
            auto few = [&](int f0, int n, int r, int first, int step, int* n_next) {
                int chunks = 0;
                if ((int)threadIdx.x < n) {
                    const KtEdge k = kt_edge(a, a.off, __ldcg(a.F[r & 1] + f0 + threadIdx.x));
                    s_e[threadIdx.x] = k.e;
                    s_pa[threadIdx.x] = k.pa;
                    s_pb[threadIdx.x] = k.pb;
                    s_na[threadIdx.x] = k.na;
                    s_nb[threadIdx.x] = k.nb;
                    chunks = (k.na + 31) >> 5;
                }
                int incl = chunks;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += y;
                }
                if (lane == 31 && warp < kKtFew / 32) s_ws[warp] = incl;
                __syncthreads();
                if (threadIdx.x < kKtFew) {
                    int before = 0;
                    for (int q = 0; q < warp; q++) before += s_ws[q];
                    s_pre[threadIdx.x] = before + incl - chunks;
                    if (threadIdx.x == kKtFew - 1) s_pre[kKtFew] = before + incl;
                }
                __syncthreads();
                const int total = s_pre[n];
                for (int c = first; c < total; c += step) {
                    int lo = 0, hi = n;   // last edge with s_pre <= c
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if (s_pre[mid] <= c) lo = mid; else hi = mid;
                    }
                    const int i = (c - s_pre[lo]) * 32 + lane;
                    if (i < s_na[lo]) probe(s_e[lo], s_pa[lo], s_pb[lo], s_nb[lo], i, r, n_next);
                    if (++beat == kKtBeat) {
                        if (lane == 0) grid_progress(&ctl->bar);
                        beat = 0;
                    }
                }
            };
            // the round is over: its counters are free for the one after next
            auto end_round = [&] {
                vc->cnt[(round + 2) % 3] = 0;
                vc->round = round + 1;
            };
            if (nf <= kKtSolo) {
                if (blockIdx.x == 0) {
                    int r = round, n = nf;
                    while (n > 0 && n <= (r == round ? kKtSolo : kKtSoloMax)) {
                        if (threadIdx.x == 0) {
                            s_next = 0;
                            grid_progress(&ctl->bar);
                        }
                        __syncthreads();
                        few(0, n, r, warp, NW, &s_next);
                        __syncthreads();
                        n = s_next;
                        r++;
                        __syncthreads();   // read before it is cleared
                    }
                    if (threadIdx.x == 0) {
                        vc->x_round = r;
                        vc->x_nf = n;
                    }
                }
                if (!sync([&] {
                        const int r = vc->x_round;
                        vc->round = r;
                        vc->cnt[r % 3] = vc->x_nf;
                        vc->cnt[(r + 1) % 3] = 0;
                        vc->cnt[(r + 2) % 3] = 0;
                    }))
                    return;
                continue;
            }
            int* const n_next = &ctl->cnt[(round + 1) % 3];
            if (nf <= kKtFew) {
                few(0, nf, round, gw, nwarps, n_next);
            } else {
                const int per = (nf + gridDim.x - 1) / gridDim.x;
                const int end = min(nf, (int)(blockIdx.x + 1) * per);
                for (int f0 = blockIdx.x * per; f0 < end; f0 += kKtFew) {
                    few(f0, min(kKtFew, end - f0), round, warp, NW, n_next);
                    __syncthreads();   // the staged edges are replaced
                    if (threadIdx.x == 0) grid_progress(&ctl->bar);
                }
            }
            if (!sync(end_round)) return;
        }
        // the edges left, and the smallest support among them
        {
            const int nL = s_nL, K = s_K, side = s_side, round = s_round;
            const int32_t* L = a.L[side];
            int32_t* L2 = a.L[side ^ 1];
            int mn = 0x7FFFFFFF;
            for (long long i0 = gt - lane; i0 < nL; i0 += nt) {
                const long long i = i0 + lane;
                const int e = i < nL ? __ldcg(L + i) : 0;
                const bool take = i < nL && __ldcg(a.state + e) == kAlive;
                const int p = warp_append(&ctl->nL2, take);
                if (take) {
                    L2[p] = e;
                    mn = min(mn, __ldcg(a.sup + e));
                }
            }
            mn = __reduce_min_sync(kFull, mn);
            if (lane == 0 && mn != 0x7FFFFFFF) atomicMin(&ctl->minsup, mn);
            if (!sync([&] {
                    const int left = vc->nL2, next = vc->minsup + 3;
                    vc->side = side ^ 1;
                    vc->nL = left;
                    vc->nL2 = 0;
                    vc->minsup = 0x7FFFFFFF;
                    vc->stop = left == 0 || 4LL * left <= a.lm;
                    if (left > 0) vc->K = next > K + 1 ? next : K + 1;
                    vc->cnt[round % 3] = 0;
                    vc->cnt[(round + 1) % 3] = 0;
                }))
                return;
            if (s_stop) return;
        }
    }
}

__global__ void k_kt_state(const unsigned char* __restrict__ alive, long long m,
                           int32_t* __restrict__ state) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m;
         e += (long long)gridDim.x * blockDim.x)
        state[e] = alive[e] ? kAlive : 0;
}

__global__ void k_kt_out(const int32_t* __restrict__ canon, const int32_t* __restrict__ truss,
                         long long m, int32_t* __restrict__ out) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m;
         e += (long long)gridDim.x * blockDim.x)
        out[e] = truss[canon[e]];
}

// Edges (in sorted-COO order) whose truss number is below K, compacted
// into an erase batch: keep[e] = truss[e] < K, pos = exclusive scan of keep.
__global__ void k_kt_below(const int32_t* __restrict__ truss, long long m, int K,
                           int32_t* __restrict__ flag) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m;
         e += (long long)gridDim.x * blockDim.x)
        flag[e] = truss[e] < K ? 1 : 0;
}

__global__ void k_kt_gather(const int32_t* __restrict__ flag, const int32_t* __restrict__ pos,
                            const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                            long long m, int32_t* __restrict__ osrc, int32_t* __restrict__ odst,
                            long long* __restrict__ total) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < m;
         e += (long long)gridDim.x * blockDim.x) {
        if (flag[e]) {
            osrc[pos[e]] = src[e];
            odst[pos[e]] = dst[e];
        }
        if (e == m - 1) *total = (long long)pos[e] + flag[e];
    }
}

int ktruss_run(hn_graph* g, int32_t* d_edge_truss) {
    cudaStream_t s = g->stream;
    const int nV = g->nV;
    const long long m = g->nE;
    if (m > 0x7FFFFFFF) throw Error(HN_ERR_INVALID, "k-truss needs nE < 2^31");
    if (m == 0) return 2;
    DevBuf<long long> off((size_t)nV + 1, s);
    DevBuf<int32_t> adj((size_t)m, s), src((size_t)m, s), canon((size_t)m, s), sup((size_t)m, s),
        truss((size_t)m, s), F((size_t)m, s), NF((size_t)m, s);
    DevBuf<unsigned char> alive((size_t)m, s), inF((size_t)m, s);
    int* cnt = (int*)g->d_scalar;  // [0] err/alive, [1] nF, [2] nNF
    export_csr64(g, off.get(), adj.get(), src.get());
    HN_CUDA(cudaMemsetAsync(cnt, 0, 4 * sizeof(int), s));
    HN_LAUNCH(k_kt_canon, grid_for(g, m, kB), kB, 0, s, off.get(), adj.get(), src.get(), m,
              canon.get(), cnt);
    read_scalars(g, 1);
    if (((int*)g->h_scalar)[0])
        throw Error(HN_ERR_INVALID, "k-truss needs a simple symmetric graph");
    HN_CUDA(cudaMemsetAsync(cnt, 0, 4 * sizeof(int), s));
    HN_CUDA(cudaMemsetAsync(inF.get(), 0, (size_t)m, s));
    const bool device_rounds = knob(kKnobKtDeviceRounds) != 0;
    DevBuf<int32_t> H;   // heavy frontier edges of each host-driven peel round
    if (!device_rounds) H.alloc((size_t)m, s);
    {
        // supports: each triangle of the degree-oriented graph credits its
        // three canonical edges once (uses the graph's scalars, so it runs
        // before the counters below are set)
        HN_CUDA(cudaMemsetAsync(sup.get(), 0, sizeof(int32_t) * (size_t)m, s));
        Oriented o;
        build_oriented(g, o, canon.get());
        edge_support(g, o, sup.get());
    }
    HN_CUDA(cudaMemsetAsync(cnt, 0, 4 * sizeof(int), s));
    HN_LAUNCH(k_kt_init, grid_for(g, m, kB), kB, 0, s, adj.get(), src.get(), m, alive.get(), cnt);
    // truss numbers start at 2 (0x02020202 per int is not 2; fill by kernel-free memset of 0
    // then write on retirement: every edge is retired exactly once)
    read_scalars(g, 1);
    long long remaining = ((int*)g->h_scalar)[0];
    int K = 3;
    int* nL = cnt + 4;      // alive-list length
    int* minsup = cnt + 5;  // smallest support on the alive list
    // the frontier of each K scans only the alive edges, and K jumps to the
    // first value that peels anything (min support + 3): R-MAT graphs reach
    // max K in the hundreds while most edges leave at small K
    DevBuf<int32_t> L((size_t)remaining + 1, s), L2((size_t)remaining + 1, s);
    auto compact = [&](const int32_t* in, long long n) {
        HN_CUDA(cudaMemsetAsync(nL, 0, sizeof(int), s));
        const int big = 0x7FFFFFFF;
        HN_CUDA(cudaMemcpyAsync(minsup, &big, sizeof(int), cudaMemcpyHostToDevice, s));
        HN_LAUNCH(k_kt_compact, grid_for(g, n, kB), kB, 0, s, in, n, alive.get(), sup.get(),
                  L2.get(), nL, minsup);
        L.swap(L2);
        HN_CUDA(cudaMemcpyAsync(g->h_scalar, cnt, 8 * sizeof(int), cudaMemcpyDeviceToHost, s));
        HN_CUDA(cudaStreamSynchronize(s));
        return ((int*)g->h_scalar)[4];
    };
    int n_alive = compact(nullptr, m);
    // the peel intersects adjacency lists; once most edges are gone the
    // lists are rebuilt from the alive edges only (hubs of the dense core
    // otherwise keep their full original lists)
    long long* loff = off.get();
    int32_t* ladj = adj.get();
    int32_t* lcanon = canon.get();
    long long lm = m;
    DevBuf<long long> coff;
    DevBuf<int32_t> cadj, ccanon, cflag, state;
    auto shrink_lists = [&]() {
        const long long keep = 2LL * n_alive;
        if (keep * 2 > lm) return;
        cflag.alloc((size_t)lm + 1, s);
        HN_CUDA(cudaMemsetAsync(cflag.get() + lm, 0, sizeof(int32_t), s));
        HN_LAUNCH(k_kt_live_pos, grid_for(g, lm, kB), kB, 0, s, (const int32_t*)lcanon, lm,
                  alive.get(), (const int32_t*)state.get(), cflag.get());
        // new slot of every live entry: an exclusive scan of the live flags;
        // a vertex's new offset is the new slot of its first old entry
        DevBuf<long long> pos((size_t)lm + 1, s), noff((size_t)nV + 1, s);
        exclusive_scan(g, (const int32_t*)cflag.get(), pos.get(), lm + 1, s);
        DevBuf<int32_t> nadj((size_t)keep + 1, s), ncanon((size_t)keep + 1, s);
        HN_LAUNCH(k_kt_shrink_off, grid_for(g, (long long)nV + 1, kB), kB, 0, s,
                  (const long long*)loff, nV, (const long long*)pos.get(), noff.get());
        HN_LAUNCH(k_kt_shrink_copy, grid_for(g, lm, kB), kB, 0, s, (const int32_t*)ladj,
                  (const int32_t*)lcanon, (const int32_t*)cflag.get(), (const long long*)pos.get(),
                  lm, nadj.get(), ncanon.get());
        coff = std::move(noff);
        cadj = std::move(nadj);
        ccanon = std::move(ncanon);
        loff = coff.get();
        ladj = cadj.get();
        lcanon = ccanon.get();
        lm = keep;
        cflag.release();
    };
    if (device_rounds) {
        // all K in cooperative launches, one between two list rebuilds
        DevBuf<KtCtl> ctl(1, s);
        state.alloc((size_t)m, s);
        HN_LAUNCH(k_kt_state, grid_for(g, m, kB), kB, 0, s, (const unsigned char*)alive.get(), m,
                  state.get());
        int round = 1;
        const int ms = ((int*)g->h_scalar)[5];
        if (ms + 3 > K) K = ms + 3;
        while (n_alive > 0) {
            KtCtl h{};
            h.round = round;
            h.nL = n_alive;
            h.K = K;
            h.minsup = INT_MAX;
            HN_CUDA(cudaMemcpyAsync(ctl.get(), &h, sizeof(KtCtl), cudaMemcpyHostToDevice, s));
            KtArgs a{ctl.get(), loff, ladj, lcanon, lm, {F.get(), NF.get()}, {L.get(), L2.get()},
                     src.get(), adj.get(), state.get(), sup.get(), truss.get(),
                     (unsigned)knob(kKnobGridWaitPolls)};
            void* args[] = {&a};
            cudaEvent_t ev = nullptr;
            if (g_profiling) profile_begin(s, &ev);
            HN_CUDA(cudaLaunchCooperativeKernel((void*)k_kt_run, dim3((unsigned)g->info.sms),
                                                dim3(kKtThreads), args, 0, s));
            if (ev) profile_end("k_kt_run", s, ev);
            count_launch();
            static_assert(sizeof(KtCtl) <= 16 * sizeof(long long), "pinned scalars");
            HN_CUDA(cudaMemcpyAsync(g->h_scalar, ctl.get(), sizeof(KtCtl), cudaMemcpyDeviceToHost,
                                    s));
            HN_CUDA(cudaStreamSynchronize(s));
            std::memcpy((void*)&h, g->h_scalar, sizeof(KtCtl));
            if (h.error) throw Error(h.error, "k-truss: a bounded wait gave up");
            if (h.side) L.swap(L2);
            n_alive = h.nL;
            K = h.K;
            round = h.round;
            if (n_alive > 0) shrink_lists();
        }
        K--;   // no edge is left at K (K = 3 on a graph without edges)
    }
    // host-driven rounds (ktruss.device_rounds = 0): launches sized to each
    // frontier, one read-back of the next frontier's size per round
    DevBuf<KtPeel> st(1, s);
    KtPeel h_peel{loff, ladj, lcanon, F.get(), NF.get(), 0, 0, 0, K, remaining, 0};
    KtPeel* h_st = &h_peel;
    if (!device_rounds)
        HN_CUDA(cudaMemcpyAsync(st.get(), h_st, sizeof(KtPeel), cudaMemcpyHostToDevice, s));
    while (!device_rounds) {
        if (remaining <= 0) { K--; break; }
        const int ms = ((int*)g->h_scalar)[5];
        if (ms + 3 > K) K = ms + 3;
        HN_LAUNCH(k_kt_begin, 1, 1, 0, s, st.get(), K);
        HN_LAUNCH(k_kt_frontier, grid_for(g, n_alive, kB), kB, 0, s, L.get(), n_alive,
                  sup.get(), alive.get(), inF.get(), st.get());
        HN_CUDA(cudaMemcpyAsync(&h_st->nf, &st.get()->nf, sizeof(int), cudaMemcpyDeviceToHost,
                                s));
        HN_CUDA(cudaStreamSynchronize(s));
        int nf = h_st->nf;
        while (nf > 0) {
            HN_LAUNCH(k_kt_peel, grid_for(g, nf, 128), 128, 0, s, st.get(), src.get(),
                      (const int32_t*)adj.get(), (const unsigned char*)alive.get(),
                      (const unsigned char*)inF.get(), sup.get(), H.get());
            HN_LAUNCH(k_kt_peel_heavy, std::min<long long>(nf, (long long)g->info.sms * 8),
                      256, 0, s, st.get(), src.get(), (const int32_t*)adj.get(),
                      (const int32_t*)H.get(), (const unsigned char*)alive.get(),
                      (const unsigned char*)inF.get(), sup.get());
            HN_LAUNCH(k_kt_retire, grid_for(g, nf, kB), kB, 0, s, (const KtPeel*)st.get(),
                      alive.get(), inF.get(), truss.get());
            HN_LAUNCH(k_kt_mark, grid_for(g, nf, kB), kB, 0, s, (const KtPeel*)st.get(),
                      inF.get());
            HN_LAUNCH(k_kt_advance, 1, 1, 0, s, st.get());
            HN_CUDA(cudaMemcpyAsync(&h_st->nf, &st.get()->nf, sizeof(int),
                                    cudaMemcpyDeviceToHost, s));
            HN_CUDA(cudaStreamSynchronize(s));
            nf = h_st->nf;
        }
        // the state comes back with the alive-list compaction's read-back
        HN_CUDA(cudaMemcpyAsync(h_st, st.get(), sizeof(KtPeel), cudaMemcpyDeviceToHost, s));
        n_alive = compact(L.get(), n_alive);
        remaining = h_st->remaining;
        if (remaining <= 0) { K--; break; }
        const long long* old_off = loff;
        shrink_lists();
        if (loff != old_off) {
            h_st->off = loff;
            h_st->adj = ladj;
            h_st->canon = lcanon;
            HN_CUDA(cudaMemcpyAsync(st.get(), h_st, 3 * sizeof(void*), cudaMemcpyHostToDevice, s));
            HN_CUDA(cudaStreamSynchronize(s));   // h_st is the copy's source
        }
        K++;
    }
    if (d_edge_truss)
        HN_LAUNCH(k_kt_out, grid_for(g, m, kB), kB, 0, s, canon.get(), truss.get(), m,
                  d_edge_truss);
    HN_CUDA(cudaStreamSynchronize(s));
    return K;
}

}  // namespace
}  // namespace hn

using namespace hn;

extern "C" int hn_ktruss(hn_graph_t* g, int32_t* max_k, int32_t* edge_truss, int mem) {
    HN_API_BEGIN
    HN_REQUIRE(g != nullptr, "graph is null");
    HN_REQUIRE(mem == HN_MEM_HOST || mem == HN_MEM_DEVICE, "bad memory kind");
    HandleUse use(g);
    HN_CUDA(cudaSetDevice(g->device));
    cudaStream_t s = g->stream;
    DevBuf<int32_t> tmp;
    int32_t* d_out = edge_truss;
    if (edge_truss && mem == HN_MEM_HOST) {
        tmp.alloc((size_t)g->nE, s);
        d_out = tmp.get();
    }
    int K = ktruss_run(g, d_out);
    if (edge_truss && mem == HN_MEM_HOST && g->nE)
        HN_CUDA(cudaMemcpyAsync(edge_truss, d_out, sizeof(int32_t) * g->nE,
                                cudaMemcpyDeviceToHost, s));
    HN_CUDA(cudaStreamSynchronize(s));
    if (max_k) *max_k = K;
    HN_API_END
}

extern "C" int hn_ktruss_keep(hn_graph_t* g, int32_t K, int32_t* max_k, int64_t* removed) {
    HN_API_BEGIN
    HN_REQUIRE(g != nullptr, "graph is null");
    HN_REQUIRE(K >= 2, "K must be at least 2");
    require_owner(g);
    std::optional<HandleUse> use;   // released before the erase call below takes it
    use.emplace(g);
    HN_CUDA(cudaSetDevice(g->device));
    cudaStream_t s = g->stream;
    if (removed) *removed = 0;
    const long long m = g->nE;
    if (m == 0) {
        if (max_k) *max_k = 2;
        return HN_OK;
    }
    DevBuf<int32_t> truss((size_t)m, s), src((size_t)m, s), dst((size_t)m, s), flag((size_t)m, s),
        pos((size_t)m, s);
    const int kmax = ktruss_run(g, truss.get());
    int rc = hn_graph_export_coo(g, 1, src.get(), dst.get(), HN_MEM_DEVICE);
    if (rc != HN_OK) return rc;
    HN_LAUNCH(k_kt_below, grid_for(g, m, kB), kB, 0, s, truss.get(), m, K, flag.get());
    exclusive_scan(g, (const int32_t*)flag.get(), pos.get(), m, s);
    DevBuf<int32_t> esrc((size_t)m, s), edst((size_t)m, s);
    long long* total = (long long*)(g->d_scalar + 6);
    HN_LAUNCH(k_kt_gather, grid_for(g, m, kB), kB, 0, s, flag.get(), pos.get(), src.get(),
              dst.get(), m, esrc.get(), edst.get(), total);
    HN_CUDA(cudaMemcpyAsync(g->h_scalar + 6, total, sizeof(long long), cudaMemcpyDeviceToHost, s));
    HN_CUDA(cudaStreamSynchronize(s));
    const long long nrem = g->h_scalar[6];
    if (max_k) *max_k = kmax;
    if (nrem == 0) return HN_OK;
    // the below-K edges leave the graph through the ordinary erase pipeline
    use.reset();
    hn_batch_t* b = nullptr;
    rc = hn_batch_create(g, nrem, esrc.get(), edst.get(), HN_MEM_DEVICE, &b);
    if (rc != HN_OK) return rc;
    int64_t n = 0;
    rc = hn_erase(g, b, HN_DEDUP_BATCH, &n);
    hn_batch_destroy(b);
    if (rc != HN_OK) return rc;
    if (removed) *removed = n;
    HN_API_END
}
