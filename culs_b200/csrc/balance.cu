// AIG balancing `b` on the GPU: the result of CULS's balancePerformV2 with
// sortDecId = 1 (src/algorithms/balance.cu:912-1382) and AIGMan::balance
// (src/aig_manager.cu:682-737), equal node for node.
//
// Every graph of a batch is worked on by a team of its own -- a block, a
// thread-block cluster, or the whole grid for one very wide graph -- that
// runs a phase from its first level to its last inside one launch: what the
// reference does with one kernel per step is a team barrier here.
//
// Phase 1, covers (k_bal_covers).  The covers (supergates) needed are those
// of the AND nodes that drive POs and of every AND leaf of a needed cover.
// Each is collected once (the DFS of localCoverTravToTable,
// balance.cu:666-751, leaves in pop order) in the order of discovery, and
// counted at its leaves.  A cover's last appear level, the longest path of
// covers from a PO, is the round in which the last cover above it was taken,
// counting down those counts.  (The reference rebuilds a frontier of all
// covers at each distance by a copy_if over all nodes, so a cover is visited
// at every level it appears on.)  A thread's DFS keeps up to 32 leaves in
// local memory; a larger cover (up to 1,024 leaves) is redone by a warp, which
// looks a literal up among the leaves 32 at a time.
//
// Phase 2, reconstruction (k_bal_rebuild).  Covers are taken deepest level
// first, in increasing node id, in chunks of 32,768 (the reference's
// iterLen): each cover's inputs (their covers' new literals, with levels)
// sorted by decreasing level then literal; then lockstep steps, one thread
// per cover, two parts per step:
//   1. the shared-node permutation and the pairing of the two lowest inputs
//      (balance.cu:113-247): a pair that is trivial or already built is
//      reused, else it is inserted into the table with id counter + cover
//      index (atomicMin keeps the smallest id of a key);
//   2. the pair's winning id, the step's largest id (the next counter), the
//      new node's level, and the pair's result put back in level order
//      (balance.cu:429-467).
// Lookups in part 1 must see the table as it was before the step: every
// entry carries the step that inserted it, and entries of the current step
// are invisible.  A level needs (its longest cover - 1) steps.
//
// Phase 3 renumbers the built nodes in id order (balance.cu:1285-1318) and
// maps the POs (balance.cu:882-910).  `b` then strashes the batch
// (AIGMan::balance with updateLevel).
//
// Bound: the latency of a step (a few dependent loads and table probes) times
// the steps of the deepest graph.  As two launches a step and four a frontier
// level, one graph after another, the 48x48 multiplier took 15.9 ms (2,671
// launches); now 3.7, of which the strash takes 0.5.
#include <algorithm>
#include <climits>
#include <numeric>
#include <vector>

#include <cooperative_groups.h>

#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace culs {

namespace {

constexpr int kBalMaxCover = 1024;  // MAX_LOCAL_COVER_SIZE, balance.cu:17
constexpr int kBalStack = 128;      // DFS_COVER_STACK_SIZE, balance.cu:18
constexpr int kBalChunk = 32768;    // iterLen, balance.cu:1125
constexpr int kBalLocal = 32;       // leaves a DFS keeps in local memory
constexpr int kBalThreads = 512;    // threads of a team's block
constexpr int kBalWarps = kBalThreads / 32;  // of a block, each with a 1,024-leaf buffer for large covers
constexpr int kBalMaxCluster = 8;   // the portable cluster size
constexpr unsigned kNoId = 0xFFFFFFFFu;
constexpr int kNoEpoch = INT_MAX;
constexpr int64_t kBalProbeCap = 1 << 20;

__device__ __forceinline__ int lit_id_(int l) { return l >> 1; }

// One graph of a group; objects, covers, leaves and table slots of the
// group's graphs lie one after another.
struct BalGraph {
    int nPIs, nPO, nObj;
    int inBase, poOff;  // first object and PO in the batch's arrays
    int obj;            // first object in the group's per-object arrays
    int flatOff;        // first leaf
    int flatCap;
    int lvOff, nLv;     // frontier levels: entries of lvCnt, lvMax, lvStart
    int tabOff;         // first table slot
    uint32_t mask;      // table slots - 1
    int outBase;        // first object of the result
    int builtOff, nBuilt;
};

// counters of a graph in the group
enum BalCount : int { kBcCnt = 0 /* round sizes, ring of 3 */, kBcBig = 3, kBcCursor, kBcLevels, kBcBuilt, kBcMaxId,
                      kBcCtr = 8 /* id counter, ring of 4 by step */, kBcMax = 12 /* largest winning id, ring of 4 */,
                      kBcFound = 16 /* covers discovered */, kBcSize = 20 };

// A built pair's table slot: the pair (lit0 << 32) | lit1, lit0 < lit1; the
// smallest id inserted with it; the step that inserted it; its level.
struct alignas(32) BalSlot {
    unsigned long long key;
    unsigned id;
    int epoch, lvl;
};

struct BalView {  // one graph: local AIGMan literals, objects [0, nObj)
    const int *F0, *F1, *PO;
    int nPIs, nPO, nObj;
};

struct BalArgs {
    const BalGraph *g;
    const int *order;  // the group's graphs, largest first
    int G;
    const int *F0, *F1, *PO;  // the batch's arrays
    int *cnt;                 // kBcSize counters per graph
    // per object of the group
    int *nfo, *drives, *pend, *lastLevel, *covLen, *covOff;
    int *found, *lists[2], *big;
    int2 *newLit;  // a cover's new {literal, level}
    int *flat;     // every collected cover's leaves
    int *scratch;  // per warp of the grid: a leaf buffer
    // per cover in processing order: (graph, last level, node id)
    const int *sorted;
    const int *lvCnt, *lvMax, *lvStart;
    int *len, *mask, *val;
    int2 *work;  // {literal, level} arrays, longest level first, at the cover's leaves' offset
    BalSlot *tab;
    int spread;  // the reconstruction deals covers by Team::spread
    int *status;
};

__device__ __forceinline__ BalView bal_view(const BalArgs &A, const BalGraph &g) {
    return BalView{A.F0 + g.inBase, A.F1 + g.inBase, A.PO + g.poOff, g.nPIs, g.nPO, g.nObj};
}

// ------------------------------------------------------------------ teams
// The threads that work on one graph together.  ld reads a word that another
// thread of the team may have written: through L1 inside a block, past it
// where the team spans several SMs.  spread: a rank that deals consecutive
// covers to different SMs of a cluster, so that the arrays of long covers share
// an L1 with as few others as possible (short ones are read together, and
// dealt by rank: 60,000 ANDs in 60 layers 4.16 ms, 4.44 by spread).  counters:
// where the graph's counters are kept while the team works on it.
struct BlockTeam {
    __device__ static int threads() { return blockDim.x; }
    __device__ static int rank() { return threadIdx.x; }
    __device__ static int spread() { return rank(); }
    __device__ static int index() { return blockIdx.x; }
    __device__ static int count() { return gridDim.x; }
    __device__ static void sync() { __syncthreads(); }
    template <class T>
    __device__ static T ld(const T *p) { return *p; }
    __device__ static int *counters(int *) {
        __shared__ int s_c[kBcSize];
        return s_c;
    }
    static constexpr bool kOwnCounters = true;
};
struct ClusterTeam {
    __device__ static int threads() { return (int)cg::this_cluster().num_threads(); }
    __device__ static int rank() { return (int)cg::this_cluster().thread_rank(); }
    __device__ static int spread() {
        return (int)(threadIdx.x * cg::this_cluster().num_blocks() + cg::this_cluster().block_rank());
    }
    __device__ static int index() { return blockIdx.x / (int)cg::this_cluster().num_blocks(); }
    __device__ static int count() { return gridDim.x / (int)cg::this_cluster().num_blocks(); }
    __device__ static void sync() { cg::this_cluster().sync(); }
    template <class T>
    __device__ static T ld(const T *p) { return __ldcg(p); }
    __device__ static int *counters(int *c) { return c; }
    static constexpr bool kOwnCounters = false;
};
struct GridTeam {
    __device__ static int threads() { return gridDim.x * blockDim.x; }
    __device__ static int rank() { return blockIdx.x * blockDim.x + threadIdx.x; }
    __device__ static int spread() { return rank(); }
    __device__ static int index() { return 0; }
    __device__ static int count() { return 1; }
    __device__ static void sync() { cg::this_grid().sync(); }
    template <class T>
    __device__ static T ld(const T *p) { return __ldcg(p); }
    __device__ static int *counters(int *c) { return c; }
    static constexpr bool kOwnCounters = false;
};

// The graph's counters for the team to work on, taken from `c` (a team
// barrier follows before they are used), and their return.
template <class Team>
__device__ __forceinline__ int *bal_open(int *c) {
    int *w = Team::counters(c);
    if (Team::kOwnCounters)
        for (int k = Team::rank(); k < kBcSize; k += Team::threads()) w[k] = c[k];
    return w;
}
template <class Team>
__device__ __forceinline__ void bal_close(int *c, const int *w) {
    if (!Team::kOwnCounters) return;
    Team::sync();
    for (int k = Team::rank(); k < kBcSize; k += Team::threads()) c[k] = w[k];
    Team::sync();
}

// The supergate DFS of localCoverTravToTable (balance.cu:666-751) into
// leaves[0..cap).  Returns the leaf count, -1 for a constant-false cover (a
// leaf and its complement), or -2 when more than cap leaves are needed.
template <class Team>
__device__ int bal_cover_dfs(const BalView &V, const int *nfo, int v, int *leaves, int cap) {
    int stk[kBalStack];
    int top = -1, n = 0;
    stk[++top] = 2 * v;
    while (top >= 0) {
        const int cur = stk[top--];
        bool same = false;
        for (int j = 0; j < n; j++) {
            const int x = leaves[j];
            if (x == cur) {
                same = true;
                break;
            }
            if (x == (cur ^ 1)) return -1;
        }
        if (same) continue;
        const int id = lit_id_(cur);
        if (cur != 2 * v && ((cur & 1) || id <= V.nPIs || Team::ld(&nfo[id]) > 1 || top + 2 >= kBalStack ||
                             n + 2 * (top + 1) + 1 >= kBalMaxCover)) {
            if (n == cap) return -2;
            leaves[n++] = cur;
            continue;
        }
        stk[++top] = V.F1[id];
        stk[++top] = V.F0[id];
    }
    return n;
}

// The same DFS by a whole warp, with room for every leaf (the DFS stops at
// 1,024): all lanes hold the walk's state, the stack lies in shared memory and
// the leaves, in global memory, are compared 32 at a time.  A thread a large
// cover, as in bal_cover_dfs, takes 4 ms for 190 leaves, a warp 0.1.  (A
// function of its own, so that the kernel's registers need not be spilled for
// it: 48x48 multiplier, which has no such cover, 1.217 ms in the kernel before
// there was this function, 1.234 with it inlined, 1.222.)
template <class Team>
__device__ __noinline__ int bal_cover_dfs_warp(BalView V, const int *nfo, int v, int *stk, int *leaves) {
    const unsigned F = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int top = 0, n = 0, cur = 2 * v;  // cur: the literal popped, with `top` left on the stack
    while (true) {
        // read at once what the literal's node may need
        const int id = lit_id_(cur), f0 = V.F0[id], f1 = V.F1[id], fanouts = Team::ld(&nfo[id]);
        bool same = false, other = false;
        for (int j = lane; j < n; j += 32) {
            const int x = leaves[j];
            same |= x == cur;
            other |= x == (cur ^ 1);
        }
        if (__any_sync(F, other)) return -1;
        if (!__any_sync(F, same)) {
            if (cur != 2 * v && ((cur & 1) || id <= V.nPIs || fanouts > 1 || top + 1 >= kBalStack ||
                                 n + 2 * top + 1 >= kBalMaxCover)) {
                if (n == kBalMaxCover) return -2;
                if (lane == 0) leaves[n] = cur;
                n++;
                __syncwarp();
            } else {
                // fanin 1 waits on the stack, fanin 0 is next
                cur = f0;
                if (lane == 0) stk[top] = f1;
                top++;
                __syncwarp();
                continue;
            }
        }
        if (top == 0) return n;
        cur = stk[--top];
        __syncwarp();  // read before the place is written again
    }
}

// Appends v to a list, one atomic per converged group of lanes.
__device__ __forceinline__ void bal_append(int *list, int *cnt, int v) {
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
    int at = 0;
    if (lane == lead) at = atomicAdd(cnt, __popc(m));
    at = __shfl_sync(m, at, lead);
    list[at + __popc(m & ((1u << lane) - 1u))] = v;
}

// Room for a cover's n leaves: its place among the graph's, n = 0 when there
// is none.
__device__ __forceinline__ int bal_take_leaves(const BalArgs &A, const BalGraph &g, int *c, int &n) {
    const int off = n > 0 ? atomicAdd(&c[kBcCursor], n) : 0;
    if (n > g.flatCap - off) {
        set_status(A.status, kDevCapacity);
        n = 0;
    }
    return off;
}

// Stores leaves first, first + step, ... of v's cover of n leaves (0: constant
// false) at place off, counts the cover at its AND leaves and lists the leaves
// found for the first time.
__device__ __forceinline__ void bal_store_cover(const BalArgs &A, const BalGraph &g, int *c, int v, const int *leaves,
                                                int n, int off, int first, int step) {
    for (int j = first; j < n; j += step) {
        A.flat[(int64_t)g.flatOff + off + j] = leaves[j];
        const int x = lit_id_(leaves[j]);
        if (x > g.nPIs && atomicAdd(&A.pend[g.obj + x], 1) == 0 && !__ldcg(&A.drives[g.obj + x]))
            bal_append(A.found + g.obj, &c[kBcFound], x);
    }
    if (first == 0) {
        A.covOff[g.obj + v] = g.flatOff + off;
        A.covLen[g.obj + v] = n;
    }
}

template <class Team>
__global__ void __launch_bounds__(kBalThreads) k_bal_covers(BalArgs A) {
    __shared__ int s_stk[kBalWarps][kBalStack];
    const int T = Team::threads(), r = Team::rank();
    for (int gi = Team::index(); gi < A.G; gi += Team::count()) {
        const BalGraph g = A.g[A.order[gi]];
        int *const c = bal_open<Team>(A.cnt + (int64_t)A.order[gi] * kBcSize);
        const BalView V = bal_view(A, g);
        int *nfo = A.nfo + g.obj, *drives = A.drives + g.obj, *pend = A.pend + g.obj, *found = A.found + g.obj,
            *big = A.big + g.obj;
        Team::sync();
        for (int v = V.nPIs + 1 + r; v < V.nObj; v += T) {
            atomicAdd(&nfo[lit_id_(V.F0[v])], 1);
            atomicAdd(&nfo[lit_id_(V.F1[v])], 1);
        }
        // the AND nodes driving POs, each once (checkCoverTravEnd, balance.cu:38-74)
        for (int k = r; k < V.nPO; k += T) {
            const int v = lit_id_(V.PO[k]);
            atomicAdd(&nfo[v], 1);
            if (v > V.nPIs && atomicExch(&drives[v], 1) == 0) bal_append(found, &c[kBcFound], v);
        }
        Team::sync();
        const int nDrive = Team::ld(&c[kBcFound]);
        // every needed cover, round by round of discovery
        for (int lo = 0, hi = nDrive; lo < hi;) {
            for (int i = lo + r; i < hi; i += T) {
                const int v = Team::ld(&found[i]);
                int leaves[kBalLocal];
                const int len = bal_cover_dfs<Team>(V, nfo, v, leaves, kBalLocal);
                if (len == -2) {
                    bal_append(big, &c[kBcBig], v);
                } else {
                    int n = max(len, 0);
                    const int off = bal_take_leaves(A, g, c, n);
                    bal_store_cover(A, g, c, v, leaves, n, off, 0, 1);
                }
            }
            Team::sync();
            const int nBig = Team::ld(&c[kBcBig]);
            if (nBig > 0) {
                const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
                int *leaves = A.scratch + ((int64_t)blockIdx.x * kBalWarps + warp) * kBalMaxCover;
                for (int i = r >> 5; i < nBig; i += T >> 5) {
                    const int v = Team::ld(&big[i]);
                    int n = bal_cover_dfs_warp<Team>(V, nfo, v, s_stk[warp], leaves);
                    if (n == -2) set_status(A.status, kDevCapacity);  // cannot happen: the DFS stops at 1,024 leaves
                    n = max(n, 0);
                    int off = 0;
                    if (lane == 0) off = bal_take_leaves(A, g, c, n);
                    n = __shfl_sync(0xffffffffu, n, 0);
                    off = __shfl_sync(0xffffffffu, off, 0);
                    bal_store_cover(A, g, c, v, leaves, n, off, lane, 32);
                    __syncwarp();  // the leaves are read before the next cover's
                }
                Team::sync();
                if (r == 0) c[kBcBig] = 0;
            }
            lo = hi;
            hi = Team::ld(&c[kBcFound]);
            Team::sync();  // read before the next round adds to it
        }
        // last appear levels: a cover is taken in the round after the last
        // cover it is a leaf of
        for (int i = r; i < nDrive; i += T) {
            const int v = Team::ld(&found[i]);
            if (Team::ld(&pend[v]) == 0) bal_append(A.lists[0] + g.obj, &c[kBcCnt], v);
        }
        Team::sync();
        int L = 0, taken = 0;
        for (int n = Team::ld(&c[kBcCnt]); n > 0; L++) {
            const int *list = A.lists[L & 1] + g.obj;
            int *next = A.lists[(L + 1) & 1] + g.obj, *nextCnt = &c[kBcCnt + (L + 1) % 3];
            if (r == 0) c[kBcCnt + (L + 2) % 3] = 0;  // read a round ago
            taken += n;
            for (int i = r; i < n; i += T) {
                const int v = Team::ld(&list[i]);
                A.lastLevel[g.obj + v] = L;
                const int len = Team::ld(&A.covLen[g.obj + v]), off = Team::ld(&A.covOff[g.obj + v]);
                for (int j = 0; j < len; j++) {
                    const int x = lit_id_(Team::ld(&A.flat[off + j]));
                    if (x > V.nPIs && atomicSub(&pend[x], 1) == 1) bal_append(next, nextCnt, x);
                }
            }
            Team::sync();
            n = Team::ld(nextCnt);
        }
        if (r == 0) {
            c[kBcLevels] = L;
            if (taken != Team::ld(&c[kBcFound])) set_status(A.status, kDevBadGraph);  // a cycle
        }
        bal_close<Team>(A.cnt + (int64_t)A.order[gi] * kBcSize, c);
    }
}

__global__ void k_bal_cover_flags(int64_t n, const int *covLen, uint8_t *flags) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) flags[p] = covLen[p] >= 0;
}

// last graph whose member `first` (increasing) is <= p
__device__ __forceinline__ int bal_graph_of(const BalGraph *g, int G, int BalGraph::*first, int p) {
    int lo = 0, hi = G - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (g[mid].*first <= p)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// per cover (in id order): its graph and last level as the sort key, its
// node's local id, and per level the cover count and the longest cover
__global__ void k_bal_cover_keys(int64_t n, const BalGraph *g, int G, int *ids, const int *lastLevel, const int *covLen,
                                 uint32_t *keys, int *lvCnt, int *lvMax) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int p = ids[i];
        const BalGraph &b = g[bal_graph_of(g, G, &BalGraph::obj, p)];
        const int k = b.lvOff + lastLevel[p];
        keys[i] = (uint32_t)k;
        ids[i] = p - b.obj;
        agg_add(lvCnt, k, 1);
        agg_max(lvMax, k, covLen[p]);
    }
}

// ------------------------------------------------------------- phase 2
struct BalTable {
    BalSlot *s;
    uint32_t mask;
    int *status;
};

__device__ __forceinline__ uint32_t bal_hash(unsigned long long k) { return (uint32_t)mix64(k); }

// insert_batch_update_min_masked (src/hash_table/hash_table.h:247-269), the
// entry tagged with the inserting step and the pair's level (the same for
// every inserter: a literal has one level).  Returns the slot, or -1; *fresh:
// the key is new.
__device__ __forceinline__ int bal_insert(const BalTable &T, unsigned long long key, unsigned id, int step, int lvl,
                                          bool *fresh) {
    uint32_t h = bal_hash(key) & T.mask;
    for (int64_t p = 0; p <= T.mask && p < kBalProbeCap; p++) {
        const unsigned long long prev = atomicCAS(&T.s[h].key, kEmptyKey, key);
        if (prev == kEmptyKey || prev == key) {
            if (prev == kEmptyKey) {
                T.s[h].epoch = step;
                T.s[h].lvl = lvl;
            }
            atomicMin(&T.s[h].id, id);
            *fresh = prev == kEmptyKey;
            return (int)h;
        }
        h = (h + 1) & T.mask;
    }
    set_status(T.status, kDevTableFull);
    return -1;
}

// Slot of a built pair as of the start of step `step` (entries of that step
// invisible) and its id, or -1.
template <class Team>
__device__ __forceinline__ int bal_find(const BalTable &T, unsigned long long key, int step, unsigned *id) {
    uint32_t h = bal_hash(key) & T.mask;
    for (int64_t p = 0; p <= T.mask && p < kBalProbeCap; p++) {
        const int4 e = Team::ld(reinterpret_cast<const int4 *>(&T.s[h]));
        const unsigned long long k = ((unsigned long long)(uint32_t)e.y << 32) | (uint32_t)e.x;
        if (k == key) {
            *id = (unsigned)e.z;
            return e.w < step ? (int)h : -1;
        }
        if (k == kEmptyKey) return -1;
        h = (h + 1) & T.mask;
    }
    set_status(T.status, kDevTableFull);
    return -1;
}

// retrieveAndNode (balance.cu:85-110): the {literal, level} of a AND b when
// it is trivial (checkTrivialAndCases, src/hash_table/hash_table.h:435-449)
// or built before `step`, else a negative literal.  AIGMan literals: 0 = TRUE,
// 1 = FALSE.
template <class Team>
__device__ __forceinline__ int2 bal_and_lookup(const BalTable &T, int2 a, int2 b, int step) {
    if (a.x == b.x) return a;
    if (a.x == (b.x ^ 1)) return make_int2(1, 0);
    if (a.x == 0) return b;
    if (b.x == 0) return a;
    if (a.x == 1 || b.x == 1) return make_int2(1, 0);
    const int l0 = min(a.x, b.x), l1 = max(a.x, b.x);
    unsigned id;
    const int h = bal_find<Team>(T, ((unsigned long long)(uint32_t)l0 << 32) | (uint32_t)l1, step, &id);
    if (h < 0) return make_int2(-1, 0);
    return make_int2((int)(id << 1), Team::ld(&T.s[h].lvl));
}

// One graph's covers of a chunk.
struct BalChunk {
    const int *covers;  // the chunk's cover roots (local ids)
    int n;
    const int *covOff;  // by node
    const int *covLen;
    int *len, *mask, *val;  // per cover: current length; step outcome (0 done, 1 new pair, 2 reused); its slot or literal
    int2 *work;
    int *c;  // the graph's counters
};

// prepareReconstructArrays (balance.cu:272-426) with sortDecId = 1: the
// inputs' new literals and levels, sorted by decreasing level, then literal.
template <class Team>
__device__ __forceinline__ void bal_prepare(const BalChunk &C, int i, const int *flat, const int2 *newLit, int nPIs) {
    const int v = C.covers[i];
    const int off = C.covOff[v], n = C.covLen[v];
    C.len[i] = n;
    int2 *a = C.work + off;
    for (int j = 0; j < n; j++) {
        const int x = flat[off + j];
        int2 e = make_int2(x, 0);
        if (lit_id_(x) > nPIs) {
            e = Team::ld(&newLit[lit_id_(x)]);
            e.x ^= x & 1;
        }
        int k = j;
        // insertion sort: (level desc, literal desc)
        while (k > 0 && (a[k - 1].y < e.y || (a[k - 1].y == e.y && a[k - 1].x < e.x))) {
            a[k] = a[k - 1];
            k--;
        }
        a[k] = e;
    }
}

// Part 1 of a step: sharedNodeDrivenPermute (balance.cu:187-247) and
// prepareDataToInsert (balance.cu:113-184), then the new pair's insertion.
// Returns whether the pair is new to the table.
template <class Team>
__device__ __forceinline__ bool bal_step1(const BalChunk &C, const BalTable &T, int i, int step, int counter) {
    const int len = C.len[i];
    if (len <= 1) {
        C.mask[i] = 0;
        return false;
    }
    int2 *a = C.work + C.covOff[C.covers[i]];
    int left = 0;
    if (len >= 3) {
        left = len - 2;
        const int border = a[left].y;
        for (left--; left >= 0 && a[left].y == border; left--) {
        }
        left++;
    }
    const int right = len - 2;
    int2 low = a[len - 2];
    const int2 last = a[len - 1];
    int2 got = make_int2(-1, 0);
    if (left < right) {
        for (int k = right; k >= left; k--) {
            const int2 e = a[k];
            got = bal_and_lookup<Team>(T, last, e, step);
            if (got.x >= 0) {
                if (e.x != low.x) {
                    a[k] = low;
                    a[right] = e;
                    low = e;
                }
                break;
            }
        }
    } else {
        got = bal_and_lookup<Team>(T, last, low, step);
    }
    C.len[i] = len - 2;
    if (got.x >= 0) {
        C.mask[i] = 2 | (got.y << 2);
        C.val[i] = got.x;
        return false;
    }
    const int l0 = min(last.x, low.x), l1 = max(last.x, low.x), lvl = max(last.y, low.y) + 1;
    bool fresh = false;
    C.mask[i] = 1 | (lvl << 2);
    C.val[i] = bal_insert(T, ((unsigned long long)(uint32_t)l0 << 32) | (uint32_t)l1, (unsigned)(counter + i), step, lvl,
                          &fresh);
    return fresh;
}

// Part 2: the winning id (retrieve_batch_masked), the step's largest id, and
// addBackLocalArrays.
template <class Team>
__device__ __forceinline__ void bal_step2(const BalChunk &C, const BalTable &T, int i, int step) {
    const int m = C.mask[i];
    if (m == 0) return;
    int lit = C.val[i];
    if ((m & 3) == 1) {
        if (lit < 0) return;  // the table is full
        const unsigned id = Team::ld(&T.s[lit].id);
        agg_max(C.c, kBcMax + (step & 3), (int)id);
        lit = (int)(id << 1);
    }
    int2 *a = C.work + C.covOff[C.covers[i]];
    const int len = C.len[i];
    bool dup = false;
    for (int j = 0; j < len && !dup; j++) dup = a[j].x == lit;
    if (dup) return;
    int k = len;
    const int2 e = make_int2(lit, m >> 2);
    while (k > 0 && e.y > a[k - 1].y) {
        a[k] = a[k - 1];
        k--;
    }
    a[k] = e;
    C.len[i] = len + 1;
}

template <class Team>
__global__ void __launch_bounds__(kBalThreads) k_bal_rebuild(BalArgs A) {
    const int T = Team::threads(), r = A.spread ? Team::spread() : Team::rank();
    for (int gi = Team::index(); gi < A.G; gi += Team::count()) {
        const BalGraph g = A.g[A.order[gi]];
        int *const c = bal_open<Team>(A.cnt + (int64_t)A.order[gi] * kBcSize);
        const BalTable H{A.tab + g.tabOff, g.mask, A.status};
        int2 *newLit = A.newLit + g.obj;
        int step = 0, built = 0, maxId = 0;
        Team::sync();
        for (int L = g.nLv - 1; L >= 0; L--) {
            const int lv = g.lvOff + L, nLv = A.lvCnt[lv], steps = A.lvMax[lv] - 1;
            for (int c0 = 0; c0 < nLv; c0 += kBalChunk) {
                const int64_t at = (int64_t)A.lvStart[lv] + c0;
                const BalChunk C{A.sorted + at, min(kBalChunk, nLv - c0), A.covOff + g.obj, A.covLen + g.obj,
                                 A.len + at,    A.mask + at,              A.val + at,       A.work,
                                 c};
                for (int i = r; i < C.n; i += T) bal_prepare<Team>(C, i, A.flat, newLit, g.nPIs);
                for (int k = 0; k < steps; k++, step++) {
                    // newIdCounter of this step; nPIs + 1 before the first (balance.cu:1167)
                    const int prev = (step - 1) & 3, top = Team::ld(&c[kBcMax + prev]);
                    const int counter = step == 0 ? g.nPIs + 1 : (top ? top + 1 : Team::ld(&c[kBcCtr + prev]));
                    if (r == 0) {
                        c[kBcCtr + (step & 3)] = counter;
                        c[kBcMax + ((step + 1) & 3)] = 0;
                        maxId = max(maxId, top);
                    }
                    for (int i = r; i < C.n; i += T) built += bal_step1<Team>(C, H, i, step, counter);
                    Team::sync();
                    for (int i = r; i < C.n; i += T) bal_step2<Team>(C, H, i, step);
                    Team::sync();
                }
                // recordReconstructedCovers (balance.cu:469-491)
                for (int i = r; i < C.n; i += T)
                    newLit[C.covers[i]] = C.len[i] == 0 ? make_int2(1, 0) : C.work[C.covOff[C.covers[i]]];
                Team::sync();
            }
        }
        built = __reduce_add_sync(0xffffffffu, built);
        if ((threadIdx.x & 31) == 0 && built) atomicAdd(&c[kBcBuilt], built);
        if (r == 0) c[kBcMaxId] = max(maxId, step ? Team::ld(&c[kBcMax + ((step - 1) & 3)]) : 0);
        bal_close<Team>(A.cnt + (int64_t)A.order[gi] * kBcSize, c);
    }
}

// ------------------------------------------------------------- phase 3
__global__ void k_bal_used(int64_t cap, const BalSlot *tab, uint8_t *flags) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; h < cap; h += stride)
        flags[h] = tab[h].key != kEmptyKey;
}

__global__ void k_bal_ids(int64_t n, const int *slots, const BalSlot *tab, uint32_t *keys) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) keys[i] = tab[slots[i]].id;
}

__global__ void k_bal_slot_graph(int64_t n, const int *slots, const BalGraph *g, int G, uint32_t *keys) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        keys[i] = (uint32_t)bal_graph_of(g, G, &BalGraph::tabOff, slots[i]);
}

// built node id -> new literal: nPIs + 1 + its rank among the graph's n built
// nodes, whose table slots in id order are `slots`
__device__ __forceinline__ int bal_out_lit(int lit, int nPIs, const BalSlot *tab, const int *slots, int n) {
    const unsigned id = (unsigned)lit_id_(lit);
    if ((int)id <= nPIs) return lit;
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (tab[slots[mid]].id < id)
            lo = mid + 1;
        else
            hi = mid;
    }
    return 2 * (nPIs + 1 + lo) + (lit & 1);
}

// nOut objects and nPO POs of the group's results, from object outFirst and
// PO poFirst of the batch on
__global__ void k_bal_out(BalArgs A, const int *slots, int64_t outFirst, int64_t nOut, int64_t poFirst, int64_t nPO,
                          int *F0n, int *F1n, int *POn) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nOut; i += stride) {
        const int p = (int)(outFirst + i);
        const BalGraph &g = A.g[bal_graph_of(A.g, A.G, &BalGraph::outBase, p)];
        const int r = p - g.outBase - 1 - g.nPIs;
        if (r < 0) {
            F0n[p] = F1n[p] = -1;
            continue;
        }
        const int *sl = slots + g.builtOff;
        const unsigned long long k = A.tab[sl[r]].key;
        F0n[p] = bal_out_lit((int)(uint32_t)(k >> 32), g.nPIs, A.tab, sl, g.nBuilt);
        F1n[p] = bal_out_lit((int)(uint32_t)k, g.nPIs, A.tab, sl, g.nBuilt);
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nPO; i += stride) {
        const int k = (int)(poFirst + i);
        const BalGraph &g = A.g[bal_graph_of(A.g, A.G, &BalGraph::poOff, k)];
        const int o = A.PO[k];
        POn[k] = lit_id_(o) <= g.nPIs
                     ? o
                     : (bal_out_lit(A.newLit[g.obj + lit_id_(o)].x, g.nPIs, A.tab, slots + g.builtOff, g.nBuilt) ^ (o & 1));
    }
}

__global__ void k_bal_init_tables(int64_t cap, BalArgs A) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; h < cap; h += stride) {
        reinterpret_cast<int4 *>(A.tab + h)[0] = make_int4(-1, -1, (int)kNoId, kNoEpoch);
    }
}

uint32_t pow2_at_least(int64_t n) {
    uint32_t c = 1024;
    while ((int64_t)c < n && c < (1u << 31)) c <<= 1;
    return c;
}

int bits_for(int64_t n) {  // bits of the values below n, at least one
    int b = 1;
    while ((1ll << b) < n) b++;
    return b;
}

// Device bytes of one graph in a group: per object 15 arrays of 4 bytes; per
// leaf (at most flatCap, in practice half of it) the leaf, its work pair,
// four 32-byte table slots and the built nodes' scratch.
int64_t bal_flat_cap(int64_t nAnd) { return 4 * nAnd + 16; }  // leaves of all covers: at most 2 per AND fanin edge visit
size_t bal_bytes(const DevGraph &d) {
    const int64_t nObj = 1 + (int64_t)d.nPIs + d.nAnds;
    return (size_t)nObj * 64 + (size_t)bal_flat_cap(d.nAnds) * 192 + 64 * 1024;
}

// How the group's graphs are worked on: one block each (clusterSize 1), a
// cluster each, or all blocks on the one graph.
struct BalTeams {
    int clusterSize, teams;
    bool grid;
    int sms;
};
// As many blocks a graph as its widest level wants threads, while every graph
// can have its team at once; a single graph wider than the largest cluster
// gets the whole grid, whose barrier costs several times a cluster's.
BalTeams bal_teams(int G, int64_t width, int sms) {
    int cluster = 1;
    while (cluster < kBalMaxCluster && cluster * kBalThreads < width && 2 * cluster * G <= sms) cluster *= 2;
    const bool grid = G == 1 && width > kBalMaxCluster * kBalThreads;
    return BalTeams{cluster, grid ? 1 : std::min(G, std::max(1, 2 * sms / cluster)), grid, sms};
}
// Runs one phase, given as its three forms.
template <class K>
cudaError_t launch_team(K block, K cluster, K all, const BalArgs &A, const BalTeams &W, cudaStream_t s) {
    if (!W.grid && W.clusterSize == 1) {
        block<<<W.teams, kBalThreads, 0, s>>>(A);
        return cudaGetLastError();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kBalThreads);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (W.grid) {
        cfg.gridDim = dim3((unsigned)W.sms);
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    } else {
        cfg.gridDim = dim3((unsigned)(W.teams * W.clusterSize));
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)W.clusterSize;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    }
    return cudaLaunchKernelEx(&cfg, W.grid ? all : cluster, A);
}

}  // namespace

// Graphs [ga, gb) of b (any of them may have no AND node); their results go to
// b's spare buffers from object ng[ga].base on, and ng's sizes and following
// bases are set.
int Engine::balance_group(const Batch &b, int ga, int gb, std::vector<DevGraph> &ng) {
    cudaStream_t s = s_;
    const int G = gb - ga;
    int rc;
    std::vector<BalGraph> bg(G);
    int64_t nObj = 0, nFlat = 0;
    size_t bytes = 0;
    int width = 1;  // nodes per level of the widest graph
    for (int i = 0; i < G; i++) {
        const DevGraph &d = b.hg[ga + i];
        BalGraph &g = bg[i];
        g = BalGraph{};
        g.nPIs = d.nPIs, g.nPO = d.nPOs, g.nObj = 1 + d.nPIs + d.nAnds;
        g.inBase = d.base, g.poOff = d.poOff;
        g.obj = (int)nObj, g.flatOff = (int)nFlat, g.flatCap = (int)bal_flat_cap(d.nAnds);
        nObj += g.nObj, nFlat += g.flatCap;
        bytes += bal_bytes(d);
        width = std::max(width, d.nAnds / std::max(d.nLevels, 1));
    }
    const BalTeams W = bal_teams(G, width, sms_);
    const size_t warps = (size_t)(W.grid ? W.sms : W.teams * W.clusterSize) * kBalWarps;
    bytes += warps * kBalMaxCover * 4 + (size_t)G * 256 + ((size_t)16 << 20);
    if ((rc = ensure_arena(bytes))) return rc;
    ar_.reset();
    std::vector<int> order(G);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return bg[x].nObj > bg[y].nObj; });
    BalArgs A{};
    BalGraph *dg = ar_.get<BalGraph>(G);
    int *dOrder = ar_.get<int>(G);
    A.cnt = ar_.get<int>((size_t)G * kBcSize);
    int *per[9];
    for (int *&p : per) p = ar_.get<int>(nObj);
    A.nfo = per[0], A.drives = per[1], A.pend = per[2], A.lastLevel = per[3], A.covLen = per[4], A.covOff = per[5];
    A.lists[0] = per[6], A.lists[1] = per[7], A.big = per[8];
    A.newLit = ar_.get<int2>(nObj);
    A.found = reinterpret_cast<int *>(A.newLit);  // discovery ends before the first new literal
    A.flat = ar_.get<int>(nFlat);
    A.scratch = ar_.get<int>(warps * kBalMaxCover);
    if (!dg || !dOrder || !A.cnt || !per[8] || !A.newLit || !A.flat || !A.scratch)
        return fail(CULS_E_OOM, "balance: arena exhausted");
    A.g = dg, A.order = dOrder, A.G = G;
    A.F0 = b.F0, A.F1 = b.F1, A.PO = b.PO;
    A.status = status_;
    check(cudaMemcpyAsync(dg, bg.data(), sizeof(BalGraph) * G, cudaMemcpyHostToDevice, s), "h2d");
    check(cudaMemcpyAsync(dOrder, order.data(), sizeof(int) * G, cudaMemcpyHostToDevice, s), "h2d");
    check(cudaMemsetAsync(A.cnt, 0, sizeof(int) * (size_t)G * kBcSize, s), "memset");
    check(cudaMemsetAsync(A.nfo, 0, sizeof(int) * nObj, s), "memset");
    check(cudaMemsetAsync(A.drives, 0, sizeof(int) * nObj, s), "memset");
    check(cudaMemsetAsync(A.pend, 0, sizeof(int) * nObj, s), "memset");
    check(cudaMemsetAsync(A.covLen, 0xFF, sizeof(int) * nObj, s), "memset");  // -1: not collected
    // ---- phase 1
    if ((rc = check(launch_team(k_bal_covers<BlockTeam>, k_bal_covers<ClusterTeam>, k_bal_covers<GridTeam>, A, W, s),
                    "balance launch")))
        return rc;
    launches_ += 1;
    // ---- covers by (graph, last level, id); per level: count and longest cover
    uint8_t *flags = ar_.get<uint8_t>(nObj);
    int *ids = ar_.get<int>(nObj), *sorted = ar_.get<int>(nObj);
    // the sort's keys, in the place of arrays that are not read any more
    uint32_t *keys = reinterpret_cast<uint32_t *>(A.lists[0]), *keys2 = reinterpret_cast<uint32_t *>(A.lists[1]);
    if (!flags || !ids || !sorted) return fail(CULS_E_OOM, "balance: arena exhausted");
    k_bal_cover_flags<<<grid_1d(nObj, kBlock, sms_ * 8), kBlock, 0, s>>>(nObj, A.covLen, flags);
    if (int e = check(compact_flags(flags, nObj, ids, counters_, ar_, s), "compact")) return e;
    std::vector<int> hc((size_t)G * kBcSize);
    check(cudaMemcpyAsync(hc.data(), A.cnt, sizeof(int) * (size_t)G * kBcSize, cudaMemcpyDeviceToHost, s), "d2h");
    if ((rc = fetch("balance covers"))) return rc;
    const int nCov = hostSmall_[0];
    // The reconstruction's teams: where covers are long on average, up to the
    // largest cluster, as their arrays and lookups outgrow the L1 of few SMs
    // (1,000 covers of 190 leaves: the call takes 35 ms with the two blocks
    // that 1,000 threads fill, 27 with eight).
    int64_t nLv = 0, nTab = 0, width2 = width;
    for (int i = 0; i < G; i++) {
        BalGraph &g = bg[i];
        const int *c = &hc[(size_t)i * kBcSize];
        const DevGraph &d = b.hg[ga + i];
        const int64_t wide = d.nAnds / std::max(d.nLevels, 1), mean = c[kBcCursor] / std::max(c[kBcFound], 1);
        width2 = std::max(width2, std::min<int64_t>(wide * (mean / kBalLocal), kBalMaxCluster * kBalThreads));
        g.lvOff = (int)nLv, g.nLv = c[kBcLevels];
        const uint32_t cap = pow2_at_least(2 * (int64_t)c[kBcCursor] + 64);
        g.tabOff = (int)nTab, g.mask = cap - 1;
        nLv += g.nLv, nTab += cap;
    }
    if (nTab > INT32_MAX) return fail(CULS_E_INVALID, "balance: tables too large");
    // ---- phase 2
    int *lvCnt = ar_.get<int>(nLv + 1), *lvMax = ar_.get<int>(nLv + 1), *lvStart = ar_.get<int>(nLv + 1);
    A.len = A.nfo, A.mask = A.drives, A.val = A.pend;  // per cover; phase 1's counts are not read any more
    A.work = ar_.get<int2>(nFlat);
    A.tab = ar_.get<BalSlot>(nTab);
    if (!lvCnt || !lvMax || !lvStart || !A.work || !A.tab) return fail(CULS_E_OOM, "balance: arena exhausted");
    check(cudaMemcpyAsync(dg, bg.data(), sizeof(BalGraph) * G, cudaMemcpyHostToDevice, s), "h2d");
    check(cudaMemsetAsync(lvCnt, 0, sizeof(int) * (nLv + 1), s), "memset");
    check(cudaMemsetAsync(lvMax, 0, sizeof(int) * (nLv + 1), s), "memset");
    if (nCov > 0) {
        k_bal_cover_keys<<<grid_1d(nCov, kBlock, sms_ * 8), kBlock, 0, s>>>(nCov, dg, G, ids, A.lastLevel, A.covLen, keys,
                                                                            lvCnt, lvMax);
        if ((rc = check(radix_sort_pairs(keys, ids, keys2, sorted, nCov, bits_for(nLv), ar_, s), "sort"))) return rc;
    }
    if (int e = check(scan_exclusive(lvCnt, lvStart, nLv, nullptr, ar_, s), "scan")) return e;
    A.sorted = sorted, A.lvCnt = lvCnt, A.lvMax = lvMax, A.lvStart = lvStart;
    k_bal_init_tables<<<grid_1d(nTab, kBlock, sms_ * 16), kBlock, 0, s>>>(nTab, A);
    A.spread = width2 > width;
    if ((rc = check(launch_team(k_bal_rebuild<BlockTeam>, k_bal_rebuild<ClusterTeam>, k_bal_rebuild<GridTeam>, A,
                                bal_teams(G, width2, sms_), s),
                    "balance launch")))
        return rc;
    launches_ += 4;
    check(cudaMemcpyAsync(hc.data(), A.cnt, sizeof(int) * (size_t)G * kBcSize, cudaMemcpyDeviceToHost, s), "d2h");
    if ((rc = fetch("balance reconstruction"))) return rc;
    // ---- phase 3: renumbering in id order
    int64_t nB = 0, out = ng[ga].base;
    int maxId = 0;
    for (int i = 0; i < G; i++) {
        BalGraph &g = bg[i];
        g.builtOff = (int)nB, g.nBuilt = hc[(size_t)i * kBcSize + kBcBuilt];
        g.outBase = (int)out;
        if (g.nBuilt > b.hg[ga + i].nAnds) return fail(CULS_E_INVALID, "balance: more nodes built than the input holds");
        maxId = std::max(maxId, hc[(size_t)i * kBcSize + kBcMaxId]);
        ng[ga + i].nAnds = g.nBuilt;
        ng[ga + i].base = g.outBase;
        nB += g.nBuilt;
        out += 1 + (int64_t)g.nPIs + g.nBuilt;
    }
    uint8_t *used = ar_.get<uint8_t>(nTab);
    int *slots = ar_.get<int>(nB + 1), *slots2 = ar_.get<int>(nB + 1);
    uint32_t *bk = ar_.get<uint32_t>(nB + 1), *bk2 = ar_.get<uint32_t>(nB + 1);
    if (!used || !slots || !slots2 || !bk || !bk2) return fail(CULS_E_OOM, "balance: arena exhausted");
    check(cudaMemcpyAsync(dg, bg.data(), sizeof(BalGraph) * G, cudaMemcpyHostToDevice, s), "h2d");
    if (nB > 0) {
        const unsigned gs = grid_1d(nB, kBlock, sms_ * 8);
        k_bal_used<<<grid_1d(nTab, kBlock, sms_ * 16), kBlock, 0, s>>>(nTab, A.tab, used);
        if (int e = check(compact_flags(used, nTab, slots, counters_, ar_, s), "compact")) return e;
        k_bal_ids<<<gs, kBlock, 0, s>>>(nB, slots, A.tab, bk);
        if ((rc = check(radix_sort_pairs(bk, slots, bk2, slots2, nB, bits_for((int64_t)maxId + 1), ar_, s), "sort")))
            return rc;
        launches_ += 2;
        if (G > 1) {
            k_bal_slot_graph<<<gs, kBlock, 0, s>>>(nB, slots2, dg, G, bk);
            if ((rc = check(radix_sort_pairs(bk, slots2, bk2, slots, nB, bits_for(G), ar_, s), "sort"))) return rc;
            launches_ += 1;
        } else {
            std::swap(slots, slots2);
        }
    }
    const int64_t poFirst = b.hg[ga].poOff, nPO = (gb < b.G ? (int64_t)b.hg[gb].poOff : b.nPO) - poFirst;
    k_bal_out<<<grid_1d(std::max(out - ng[ga].base, nPO), kBlock, sms_ * 8), kBlock, 0, s>>>(
        A, slots, ng[ga].base, out - ng[ga].base, poFirst, nPO, b.F0s, b.F1s, b.POs);
    launches_ += 1;
    if (gb < b.G) ng[gb].base = (int)out;
    return check(cudaGetLastError(), "balance launch");
}

// AIGMan::balance(sortDecId = 1) over every graph of b.
int Engine::balance(Batch &b, bool updateLevel) {
    b.keep = false;  // prevCmdRewrite = 0 (aig_manager.cu:729)
    if (!b.pool) b.pool = pool_;
    int rc;
    if ((rc = check(b.reserve_spare(b.nObj + 1, b.nPO + 1), "cudaMalloc"))) return rc;
    std::vector<DevGraph> ng = b.hg;
    // Groups of graphs: together up to what the largest alone needs, or a
    // sixteenth of the HBM budget -- a batch needs no more scratch than its
    // largest graph unless there is plenty.
    size_t cap = budget_ / 16;
    for (const DevGraph &d : b.hg) cap = std::max(cap, bal_bytes(d));
    if (b.G > 0) ng[0].base = 0;
    for (int ga = 0; ga < b.G;) {
        size_t bytes = bal_bytes(b.hg[ga]);
        int gb = ga + 1;
        while (gb < b.G && bytes + bal_bytes(b.hg[gb]) <= cap) bytes += bal_bytes(b.hg[gb++]);
        rc = balance_group(b, ga, gb, ng);
        if ((rc == CULS_E_OOM || rc == CULS_E_BUDGET) && gb - ga > 1) {
            cap = 0;  // one graph at a time
            continue;
        }
        if (rc) return rc;
        ga = gb;
    }
    if ((rc = fetch("balance output"))) return rc;
    ar_.reset();
    const int64_t nObj = b.G > 0 ? (int64_t)ng[b.G - 1].base + 1 + ng[b.G - 1].nPIs + ng[b.G - 1].nAnds : 0;
    if ((rc = check(cudaMemcpyAsync(b.dg, ng.data(), sizeof(DevGraph) * b.G, cudaMemcpyHostToDevice, s_), "h2d")))
        return rc;
    if ((rc = sync())) return rc;
    b.swap_spare();
    b.hg = ng;
    b.nObj = nObj;
    // levels: a strash (the `b` command), else the depth as read
    return updateLevel ? st(b, false) : batch_depth(b);
}

}  // namespace culs
