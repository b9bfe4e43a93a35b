// Existence table and per-node evaluation: BuildHashTable + EvaluateNode
// (CULS src/algorithms/rewrite.cu:378-471).  The chained table of the
// reference becomes an open-addressing table on 64-bit CAS keys (fanin0 id,
// fanin1 id, compl0, compl1) with one region per graph.  Both the build and
// the evaluation visit the nodes graph by graph (the front's byGraph order),
// so the region, cuts and fanin arrays a block touches belong to the few
// graphs in flight.
//
// Evaluation works on (node, cut) items, and walks a class's library forest
// only for those whose inputs' filters leave a root open (see k_evaluate).
#include <algorithm>
#include <vector>

#include "rw_work.cuh"

namespace culs {

namespace {

constexpr int kEvalBlock = 64;
// Resident blocks an SM: at 56 registers a thread 16 fit.  256 graphs of up to
// 200k ANDs: 8.8 ms with 12, 7.5 with 16, 7.7 with 20.
constexpr int kEvalBlocksPerSm = 16;

__global__ void k_table_clear(int64_t n, TabSlot *slots) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        reinterpret_cast<int4 *>(slots)[i] = make_int4(-1, -1, 0x7FFFFFFF, 0);
}

// Inserts the AND nodes at graph-major indices [lo, hi) of byGraph.
__global__ void k_table_build(int64_t nL0, int64_t lo, int64_t hi, const int *byGraph, const int *w0, const int *w1,
                              const int *wg, const DevGraph *dg, RegionTable tab, unsigned long long *pairs,
                              int *status) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = lo + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < hi; i += stride) {
        const int q = byGraph[i];
        if (q < nL0) continue;  // constant or PI
        int f0 = w0[q], f1 = w1[q];
        const int g = wg[q];
        int cp = dg[g].cpos;
        // rewrite.cu:454 skips nodes whose fanins are both the constant
        if ((f0 >> 1) == cp && (f1 >> 1) == cp) continue;
        region_insert(table_region(tab, g), and_key(f0 >> 1, f1 >> 1, f0 & 1, f1 & 1), q, status);
        if ((f0 >> 1) <= (f1 >> 1))  // others no lookup finds
            atomicOr(&pairs[f1 >> 1], 1ull << (pair_bit(f0 >> 1) + 2 * (f0 & 1) + (f1 & 1)));
    }
}

struct EvalArgs {
    int64_t nL0, lo, hi;  // evaluates the nodes at graph-major indices [lo, hi) of byGraph
    const int *byGraph;
    EvalIn E;
    RegionTable tab;
    const int4 *cutL;
    const int2 *cutM;
    const int *wg;
    const DevGraph *dg;
    int useZeros;
    int *mffcNodes;  // per warp of the grid, per item: up to 8 MFFC node positions
    int8_t *bestCut;
    uint8_t *bestOut;
    uint8_t *candFlag;
};

// Per-warp shared state of k_evaluate: lists of the slots (local node * 8 +
// cut slot) of the warp's nodes, and one result per slot.
constexpr int kWarpNodes = 32;
struct WarpItems {
    uint16_t item[kWarpNodes * 8];  // the evaluable cuts; then those that still need the walk
    uint16_t full[kWarpNodes * 8];  // those whose MFFC needs the full traversal
    int2 res[kWarpNodes * 8];       // {gain * 16 + root index, level} or {-1, 0}
    uint16_t roots[kWarpNodes * 8];  // open_roots
    uint8_t saved[kWarpNodes * 8];  // CalcMFFC's count
    uint8_t nDel[kWarpNodes * 8];   // its MFFC nodes (in EvalArgs::mffcNodes)
};

struct EvalItem {
    int q, g, cpos;
    uint32_t pk;
    int4 l;
};

__device__ __forceinline__ EvalItem eval_item(const EvalArgs &A, int64_t base, int slot) {
    EvalItem x;
    x.q = A.byGraph[base + (slot >> 3)];
    x.g = A.wg[x.q];
    x.cpos = A.dg[x.g].cpos;
    const int64_t idx = (int64_t)x.q * 8 + (slot & 7);
    x.pk = (uint32_t)A.cutM[idx].y;
    x.l = A.cutL[idx];
    return x;
}

// Appends slot to list (n entries so far) for the lanes that keep theirs.
__device__ __forceinline__ int append(uint16_t *list, int n, bool keep, int slot, int lane) {
    const unsigned b = __ballot_sync(0xffffffffu, keep);
    if (keep) list[n + __popc(b & ((1u << lane) - 1u))] = (uint16_t)slot;
    return n + __popc(b);
}

// A warp takes 32 consecutive nodes of the graph-major order and sieves their
// cuts, 32 items at a time and every list dense again after each step: the
// evaluable cuts (about half of the slots), the MFFC traversal of those that
// need one (a quarter), and the walk through the cones of the roots that
// open_roots leaves.  Each lane then folds its own node's results in slot
// order, the order of the reference's loop.  Warps never wait for one another.
//
// Bound by the walks' chains of dependent loads (three quarters of a warp's
// time).  Walking the whole forest for every cut, cuts sorted by class so that
// lanes walk forests of like depth, with the matches in shared memory (16
// warps an SM): 13.3 ms for 256 graphs of up to 200k ANDs, 1.36 for a 1M-AND
// layered graph; reached nodes only: 11.4 and 1.23; without the sort, 32 warps:
// 7.6 and 0.81; open roots only: 7.4 and 0.81.  One probe a step for all lanes
// of a warp: 7.7 and 0.84, as 2 of 6 roots are open on average and the lanes'
// walks are short.
__global__ void __launch_bounds__(kEvalBlock, kEvalBlocksPerSm) k_evaluate(EvalArgs A) {
    __shared__ WarpItems s_w[kEvalBlock / 32];
    const int lane = threadIdx.x & 31;
    WarpItems &W = s_w[threadIdx.x >> 5];
    const int64_t nWarpChunks = (A.hi - A.lo + kWarpNodes - 1) / kWarpNodes;
    const int64_t warp = (int64_t)blockIdx.x * (kEvalBlock / 32) + (threadIdx.x >> 5);
    const int64_t warpStride = (int64_t)gridDim.x * (kEvalBlock / 32);
    int *const mffcNodes = A.mffcNodes + warp * (kWarpNodes * 8 * 8);
    const int least = A.useZeros ? 0 : 1;
    for (int64_t wc = warp; wc < nWarpChunks; wc += warpStride) {
        const int64_t base = A.lo + wc * kWarpNodes;
        // 1. the evaluable cuts; a node's 8 slots lie side by side
        const int q = base + lane < A.hi ? A.byGraph[base + lane] : -1;
        int nItems = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int slot = k * 32 + lane, nq = __shfl_sync(0xffffffffu, q, slot >> 3);
            bool use = false;
            if (nq >= A.nL0) {  // not the constant, a PI or past the end
                const uint32_t pk = (uint32_t)A.cutM[(int64_t)nq * 8 + (slot & 7)].y;
                use = packed_used(pk) && packed_nleaves(pk) >= 3;
            }
            W.res[slot] = make_int2(-1, 0);
            nItems = append(W.item, nItems, use, slot, lane);
        }
        __syncwarp();
        // 2. the items whose MFFC is the root alone (nothing deleted): most
        // end here.  Entries kept in item lie before those read.
        int nFull = 0, nWalk = 0;
        for (int it0 = 0; it0 < nItems; it0 += 32) {
            const int slot = it0 + lane < nItems ? W.item[it0 + lane] : -1;
            bool full = false, walk = false;
            if (slot >= 0) {
                const EvalItem x = eval_item(A, base, slot);
                const int leaves[4] = {x.l.x, x.l.y, x.l.z, packed_nleaves(x.pk) == 3 ? x.cpos : x.l.w};
                full = !mffc_trivial(A.E, x.q, leaves);
                if (!full) {
                    const uint32_t roots = open_roots(A.E, cut_view(A.E, x.cpos, x.pk, x.l), 1 - least);
                    walk = roots != 0;
                    W.roots[slot] = (uint16_t)roots;
                    W.saved[slot] = 1;
                    W.nDel[slot] = 0;
                }
            }
            __syncwarp();
            nFull = append(W.full, nFull, full, slot, lane);
            nWalk = append(W.item, nWalk, walk, slot, lane);
        }
        __syncwarp();
        // 3. the others' MFFCs
        for (int k0 = 0; k0 < nFull; k0 += 32) {
            const int slot = k0 + lane < nFull ? W.full[k0 + lane] : -1;
            bool walk = false;
            if (slot >= 0) {
                const EvalItem x = eval_item(A, base, slot);
                const int leaves[4] = {x.l.x, x.l.y, x.l.z, packed_nleaves(x.pk) == 3 ? x.cpos : x.l.w};
                int n;
                const int saved = mffc_size(A.E, x.q, leaves, mffcNodes + slot * 8, &n);
                const uint32_t roots = open_roots(A.E, cut_view(A.E, x.cpos, x.pk, x.l), saved - least);
                walk = roots != 0;
                W.roots[slot] = (uint16_t)roots;
                W.saved[slot] = (uint8_t)saved;
                W.nDel[slot] = (uint8_t)n;
            }
            nWalk = append(W.item, nWalk, walk, slot, lane);
        }
        __syncwarp();
        // 4. the walks
        for (int it = lane; it < nWalk; it += 32) {
            const int slot = W.item[it];
            const EvalItem x = eval_item(A, base, slot);
            EvalIn E = A.E;
            E.tab = table_region(A.tab, x.g);
            const CutBest b = eval_cut(E, x.q, cut_view(E, x.cpos, x.pk, x.l), W.roots[slot], least, W.saved[slot],
                                       W.nDel[slot], mffcNodes + slot * 8);
            if (b.out >= 0) W.res[slot] = make_int2(b.gain * 16 + b.out, b.level);
        }
        __syncwarp();
        // 5. fold this lane's node's cuts in slot order
        if (q >= A.nL0) {
            int bc = -1, bo = -1, gain = 0, level = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const int2 r = W.res[lane * 8 + k];
                if (r.x >= 0) fold_cut_best(CutBest{r.x >> 4, r.y, r.x & 15}, k, bc, bo, gain, level);
            }
            A.bestCut[q] = (int8_t)bc;
            A.bestOut[q] = (uint8_t)(bo < 0 ? 0 : bo);
            A.candFlag[q] = bc >= 0;
        }
        __syncwarp();
    }
}

}  // namespace

int rw_evaluate(ExecCtx &X, RwWork &w, const Batch &b) {
    const int64_t N = w.N;
    cudaStream_t s = X.s;
    int64_t nAnd = N - w.nL0;
    // region of graph g: 4 * its AND count + 8 slots.  At load factor <= 1/4
    // a linear probe ends in its home slot for ~80% of misses and ~90% of
    // hits (at 1/2 a miss scans 2.5 slots on average), and every extra slot
    // is a dependent load the whole warp waits for.
    std::vector<int64_t> off(w.G + 1);
    off[0] = 0;
    for (int g = 0; g < w.G; g++) off[g + 1] = off[g] + 4 * (int64_t)b.hg[g].nAnds + 8;
    const int64_t nSlots = off[w.G];
    TabSlot *slots = X.ar->get<TabSlot>(nSlots);
    int64_t *dOff = X.ar->get<int64_t>(w.G + 1);
    w.bestCut = X.ar->get<int8_t>(N);
    w.bestOut = X.ar->get<uint8_t>(N);
    uint8_t *candFlag = X.ar->get<uint8_t>(N);
    w.cand = X.ar->get<int>(N);
    // one resident wave; a second wave of a grid-stride kernel would only start as the first ends
    const unsigned evalGrid = grid_1d(N, kEvalBlock, X.sms * kEvalBlocksPerSm);
    int *mffcNodes = X.ar->get<int>((size_t)evalGrid * (kEvalBlock / 32) * kWarpNodes * 8 * 8);
    const size_t kept = X.ar->used();
    unsigned long long *pairs = X.ar->get<unsigned long long>(N);
    if (!slots || !dOff || !w.bestCut || !w.bestOut || !candFlag || !w.cand || !mffcNodes || !pairs)
        return X.fail(CULS_E_OOM, "rw: scratch arena exhausted (table)");
    w.tab = RegionTable{slots, dOff};
    int rc;
    if ((rc = X.check(cudaMemcpyAsync(dOff, off.data(), sizeof(int64_t) * (w.G + 1), cudaMemcpyHostToDevice, s),
                      "h2d")))
        return rc;
    if ((rc = X.check(cudaMemsetAsync(w.bestCut, 0xFF, N, s), "memset"))) return rc;
    if ((rc = X.check(cudaMemsetAsync(candFlag, 0, N, s), "memset"))) return rc;
    if ((rc = X.check(cudaMemsetAsync(pairs, 0, sizeof *pairs * N, s), "memset"))) return rc;
    if (nAnd > 0) {
        k_table_clear<<<X.grid(nSlots), kBlock, 0, s>>>(nSlots, slots);
        X.mark(kMkEvalK0);
        // Graphs in groups of at most kGroupSlots table slots (16M by
        // default: 256 MB of regions; a tuned parameter), each group's
        // regions built right before its nodes are evaluated, so that more of
        // the probes find them in L2 (a single larger graph is a group of its
        // own).  Small groups leave the GPU idle at their ends, large ones
        // outgrow L2: 256 graphs of up to 200k ANDs 9.3 ms with 1M slots, 7.4
        // with 4M, 7.3 with 8M, 7.5 with 16M, 7.9 with 64M; 128 of up to 100k
        // 2.33, 1.94, 1.91, 1.89, 1.89; 2,000 of up to 2k 1.10, 0.97, 0.90,
        // 0.90, 0.91.
        const int64_t kGroupSlots = (int64_t)X.tune->evalGroupMSlots << 20;
        int g0 = 0;
        while (g0 < w.G) {
            int g1 = g0 + 1;
            while (g1 < w.G && off[g1 + 1] - off[g0] <= kGroupSlots) g1++;
            const int64_t lo = b.hg[g0].base, hi = g1 < w.G ? (int64_t)b.hg[g1].base : N;
            k_table_build<<<X.grid(hi - lo), kBlock, 0, s>>>(w.nL0, lo, hi, w.byGraph, w.w0, w.w1, w.wg,
                                                             w.dg, w.tab, pairs, X.status);
            EvalArgs A{w.nL0,  lo,     hi,     w.byGraph,
                       EvalIn{w.w0, w.w1, w.ref, w.wlev, X.lib, TabRegion{}, pairs, X.status},
                       w.tab,  w.cutL, w.cutM, w.wg,      w.dg,
                       w.useZeros ? 1 : 0, mffcNodes, w.bestCut, w.bestOut, candFlag};
            const unsigned grid = std::min(evalGrid, X.grid(hi - lo, kEvalBlock));
            k_evaluate<<<grid, kEvalBlock, 0, s>>>(A);
            X.launched(2);
            g0 = g1;
        }
        X.mark(kMkEvalK1);
        X.launched(1);
    }
    X.ar->release(kept);  // the filters end here; what reuses their room comes later on this stream
    if ((rc = X.check(compact_flags(candFlag, N, w.cand, X.counters + 8, *X.ar, s), "compact"))) return rc;
    if ((rc = X.fetch("rw evaluate"))) return rc;
    w.nCand = X.hostSmall[8];
    return 0;
}

}  // namespace culs
