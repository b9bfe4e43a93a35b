// Structural hashing with dangling-node removal (`st`, and the
// deduplication that ends `rw`): a B200 restatement of Aig::strash (CULS
// src/aig/strash.cu:190-314) and of the CPU variants (src/aig/strash.cu:
// 322-466, src/aig_manager.cu:454-522).
//
// Reference semantics kept:
//  * dangling AND nodes are those outside the transitive fanin of the POs
//    (the fix-point of markDanglingNodesIter, strash.cu:175-188);
//  * nodes are hashed frontier by frontier, where a node's frontier is its
//    ASAP level among the remaining nodes, and inside a frontier in id order
//    (strash.cu:247-277);
//  * fanins are mapped to new literals, sorted, folded by
//    checkTrivialAndCases (src/hash_table/hash_table.h:435-449), then hashed
//    on the 64-bit key (lit0 << 32 | lit1) (hash_table.h:427-433);
//  * survivors are renumbered consecutively in (frontier, id) order and the
//    frontier count becomes the AIG level (strash.cu:279-300,483).
// Deterministic choice: among equal keys the earliest node in (frontier, id)
// order wins (the reference keeps whichever insertion lands first).
//
// B200 design: no per-frontier host loop.  Liveness is a reverse Kahn
// worklist, levels an in-order dataflow (a forward Kahn worklist over a
// fanout CSR as the fallback; a single graph of up to 57,000 nodes in one
// block's shared memory), and hashing either rounds that iterate the mapping
// to its fixed point, the first over all nodes and the later ones over those
// whose fanins' mapping changed (batches of up to 16M live nodes), or a single
// in-order dataflow pass whose dependency waits are per-level completion
// counters (bounded spins).
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "kernels.cuh"
#include "levels.cuh"
#include "rw_work.cuh"
#include "sched.cuh"

namespace culs {

namespace {

__device__ __forceinline__ bool is_and(const int *L0, int v) { return L0[v] >= 0; }

__global__ void k_fanout_count(int64_t M, const int *L0, const int *L1, const int *po, int64_t nPO, int *cnt) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < M; v += stride) {
        int a = L0[v];
        if (a < 0) continue;
        atomicAdd(&cnt[a >> 1], 1);
        atomicAdd(&cnt[L1[v] >> 1], 1);
    }
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nPO; k += stride) atomicAdd(&cnt[po[k] >> 1], 1);
}

__global__ void k_dead_seed_flags(int64_t M, const int *L0, const int *cnt, uint8_t *flags) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < M; v += stride)
        flags[v] = (L0[v] >= 0 && cnt[v] == 0) ? 1 : 0;
}

// Reverse Kahn: a node whose fanout count reaches zero is dangling.
__global__ void __launch_bounds__(kBlock) k_dead_queue(WorkQueue q, const int *L0, const int *L1, int *cnt,
                                                        uint8_t *dead, int *status) {
    int h = -1;
    bool fin = false;
    int64_t idle = 0;
    while (true) {
        const int v = queue_try_pop_warp(q, h, fin);
        int p0 = -1, p1 = -1;
        if (v >= 0) {
            dead[v] = 1;
            int u0 = L0[v] >> 1, u1 = L1[v] >> 1;
            if (L0[u0] >= 0 && atomicSub(&cnt[u0], 1) == 1) p0 = u0;
            if (L0[u1] >= 0 && atomicSub(&cnt[u1], 1) == 1) p1 = u1;
        }
        queue_push_warp(q, p0);
        queue_push_warp(q, p1);
        queue_done_warp(q, v >= 0);
        if (queue_round_end(fin, v >= 0, idle, status)) break;
    }
}

// level[v] = 1 for a live AND node without AND fanins (the seeds), -1 for the
// other AND nodes, 0 for the constant and PIs; outdeg[u] = live AND fanouts
// (a node whose two fanins are one node counts once).
__global__ void k_live_degrees(int64_t M, const int *L0, const int *L1, const uint8_t *dead, int *level, int *outdeg,
                               uint8_t *liveFlag, uint8_t *seedFlag) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < M; v += stride) {
        int a = L0[v];
        bool live = a >= 0 && !dead[v];
        liveFlag[v] = live;
        int pend = 0;
        if (live) {
            int u0 = a >> 1, u1 = L1[v] >> 1;
            if (L0[u0] >= 0) {
                pend++;
                atomicAdd(&outdeg[u0], 1);
            }
            if (L0[u1] >= 0 && u1 != u0) {
                pend++;
                atomicAdd(&outdeg[u1], 1);
            }
        }
        level[v] = a < 0 ? 0 : (live && pend == 0 ? 1 : -1);
        seedFlag[v] = live && pend == 0;
    }
}

__global__ void k_csr_fill(int64_t M, const int *L0, const int *L1, const uint8_t *liveFlag, int *cursor, int *adj) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < M; v += stride) {
        if (!liveFlag[v]) continue;
        int u0 = L0[v] >> 1, u1 = L1[v] >> 1;
        if (L0[u0] >= 0) adj[atomicAdd(&cursor[u0], 1)] = (int)v;
        if (L0[u1] >= 0 && u1 != u0) adj[atomicAdd(&cursor[u1], 1)] = (int)v;
    }
}

// Level-synchronous Kahn: ASAP level of every live AND node (PIs and
// constant: 0), one launch per level.  The queue's levels are consecutive
// segments of `items`; launch L reads its segment's start and size from a
// three-slot ring (written by launch L - 1, which has finished), releases
// the fanouts of every node of level L, and appends to level L + 1's
// segment each fanout whose other fanin finished earlier (no pending
// counters: a node's level is written when it is appended, so the levels up
// to L are all known when launch L starts, and of two fanins on the same
// level the one at the higher position appends).  Thread 0 of block 0
// sets the next segment's start and clears the slot that launch L + 1 will
// append to, which no other block of launch L touches.  No thread waits on
// another.  ring[0..2]: segment sizes, ring[3..5]: segment starts, both by
// level mod 3.
__global__ void __launch_bounds__(kBlock) k_level_step(int L, int *items, int *ring, const int *off, const int *adj,
                                                        const int *L0, const int *L1, int *level, const int *gid,
                                                        int *graphLevels, int *maxLevel) {
    const int r = L % 3;
    const int start = ring[3 + r], n = ring[r];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        ring[3 + (L + 1) % 3] = start + n;
        ring[(L + 2) % 3] = 0;
        if (n > 0) atomicMax(maxLevel, L);
    }
    if (n == 0) return;
    int *nextCnt = ring + (L + 1) % 3;
    const int nextBase = start + n;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; i0 < n; i0 += warps * 32) {
        const int64_t i = i0 + lane;
        int k = 0, e = 0, v = -1;
        if (i < n) {
            v = items[start + i];
            agg_max(graphLevels, gid[v], L);
            k = off[v];
            e = off[v + 1];
        }
        // release the fanouts, one fanout per lane per round: v pushes w when
        // w's other fanin is not an AND node, is below level L, or is on
        // level L at a lower position (levels up to L are all set when the
        // launch starts; later ones read as -1 or L + 1)
        while (__any_sync(0xffffffffu, k < e)) {
            bool push = false;
            int w = 0;
            if (k < e) {
                w = adj[k++];
                const int a = L0[w] >> 1, b = L1[w] >> 1;
                const int u = a == v ? b : a;
                if (u == v || L0[u] < 0) {
                    push = true;
                } else {
                    const int lu = level[u];
                    push = lu >= 0 && (lu < L || (lu == L && u < v));
                }
                if (push) level[w] = L + 1;
            }
            const unsigned b = __ballot_sync(0xffffffffu, push);
            if (b) {
                int base = 0;
                if (lane == 0) base = atomicAdd(nextCnt, __popc(b));
                base = __shfl_sync(0xffffffffu, base, 0);
                if (push) items[nextBase + base + __popc(b & ((1u << lane) - 1u))] = w;
            }
        }
    }
}

// done: 0 until an AND node's level is known, then level + 1
__global__ void k_live_flags(int64_t M, const int *L0, const uint8_t *dead, uint8_t *liveFlag, int *done) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < M; v += stride) {
        const bool isAnd = L0[v] >= 0;
        liveFlag[v] = isAnd && !dead[v];
        done[v] = isAnd ? 0 : 1;
    }
}

// Levels of a graph-major batch whose positions are topological (`st`):
// the in-order dataflow of the rw front over the interleaved chunk schedule
// (sched.cuh), instead of a worklist over a fanout CSR.  Every AND node gets
// its ASAP level; only live nodes count towards a graph's depth.  A node's
// level + 1 in done[] is the one word its fanouts wait on and read.
__global__ void __launch_bounds__(kBlock) k_st_levelize(ChunkSched S, const int *L0, const int *L1,
                                                         const uint8_t *liveFlag, const int *gid, int *level,
                                                         int *done, int *graphLevels, int *counter, int *maxLevel,
                                                         int *status) {
    __shared__ int64_t s_begin, s_end;
    int myMax = 0;
    while (true) {
        if (threadIdx.x == 0) {
            const int64_t c = atomicAdd(counter, 1);
            if (c < S.total) {
                sched_chunk(S, c, s_begin, s_end);
            } else {
                s_begin = s_end = -1;
            }
        }
        __syncthreads();
        const int64_t begin = s_begin, end = s_end;
        __syncthreads();
        if (begin < 0) break;
        const int64_t p = begin + threadIdx.x;
        if (p >= end) continue;
        const int a = L0[p];
        if (a < 0) continue;  // constant or PI: level 0, done preset
        const int u0 = a >> 1, u1 = L1[p] >> 1;
        int d0, d1;
        if (!wait_words(&done[u0], &done[u1], 1, status, &d0, &d1)) continue;
        const int lv = d0 > d1 ? d0 : d1;
        st_relaxed(&done[p], lv + 1);
        __stcg(&level[p], lv);
        if (liveFlag[p]) {
            agg_max(graphLevels, gid[p], lv);
            myMax = lv > myMax ? lv : myMax;
        }
    }
    // every thread of the block leaves the loop at the same claim
    myMax = __reduce_max_sync(0xffffffffu, myMax);
    if ((threadIdx.x & 31) == 0 && myMax > 0) atomicMax(maxLevel, myMax);
}

// Levels over an order that is topological up to a few fanins placed later
// (the rewrite's deduplication: see k_proc_order).  A pass runs the nodes of
// `list` in order; a node waits only for AND fanins earlier in the order.  A
// fanin later in the order that is not done yet, or one left unresolved,
// leaves the node unresolved (done = 2), and the unresolved nodes form the
// next pass's list.  Every wait is on a node whose chunk was claimed
// earlier, so no pass can deadlock, and each pass resolves at least the
// unresolved nodes whose fanins are all resolved.  done[] is the word a node
// publishes: 0 pending, 2 unresolved, level + 2 once resolved.
__global__ void __launch_bounds__(kBlock) k_order_levelize(int64_t n, const int *list, const int *posOf, const int *L0,
                                                            const int *L1, const uint8_t *liveFlag, const int *gid,
                                                            int *level, int *done, int *graphLevels, int *counter,
                                                            int *maxLevel, int *status) {
    __shared__ int64_t s_begin;
    int myMax = 0;
    const int64_t nChunks = (n + kBlock - 1) / kBlock;
    while (true) {
        if (threadIdx.x == 0) {
            const int64_t c = atomicAdd(counter, 1);
            s_begin = c < nChunks ? c * kBlock : -1;
        }
        __syncthreads();
        const int64_t begin = s_begin;
        __syncthreads();
        if (begin < 0) break;
        const int64_t i = begin + threadIdx.x;
        if (i >= n) continue;
        const int v = list[i];
        if (v < 0 || !liveFlag[v]) continue;
        const int pv = posOf[v];
        int lv = 0;
        bool ok = true;
        for (int k = 0; k < 2 && ok; k++) {
            const int u = (k == 0 ? L0[v] : L1[v]) >> 1;
            if (L0[u] < 0) continue;  // constant or PI: level 0
            int d = ld_relaxed(&done[u]);
            if (d == 0 && posOf[u] < pv && !wait_word(&done[u], 1, status, &d)) {
                ok = false;
                break;
            }
            if (d < 3) {  // pending behind this node in the order, or unresolved
                ok = false;
                break;
            }
            const int l = d - 2;
            lv = l > lv ? l : lv;
        }
        if (!ok) {
            st_relaxed(&done[v], 2);
            continue;
        }
        lv += 1;
        st_relaxed(&done[v], lv + 2);
        __stcg(&level[v], lv);
        agg_max(graphLevels, gid[v], lv);
        myMax = lv > myMax ? lv : myMax;
    }
    myMax = __reduce_max_sync(0xffffffffu, myMax);
    if ((threadIdx.x & 31) == 0 && myMax > 0) atomicMax(maxLevel, myMax);
}

// The same order as levels_block takes it: order index k's fanins as literals
// over order indexes.
__global__ void k_order_fanins(int64_t n, const int *list, const int *posOf, const int *L0, const int *L1,
                               const uint8_t *liveFlag, int *a0, int *a1) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        const int v = list[k];
        const int a = v >= 0 ? L0[v] : 0;
        if (v < 0 || a < 0 || !liveFlag[v]) {
            a0[k] = v >= 0 && a < 0 ? kLevelZero : kLevelSkip;
            continue;
        }
        const int b = L1[v];
        a0[k] = 2 * posOf[a >> 1] + (a & 1);
        a1[k] = 2 * posOf[b >> 1] + (b & 1);
    }
}

__global__ void k_unresolved_flags(int64_t n, const int *list, const int *done, uint8_t *flag) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int v = list[i];
        flag[i] = v >= 0 && done[v] == 2;
    }
}

// next list = list[idx[k]], reset to pending
__global__ void k_unresolved_next(int64_t n, const int *idx, const int *list, int *next, int *done) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        const int v = list[idx[k]];
        next[k] = v;
        done[v] = 0;
    }
}

// lvlCnt has nBins counters (levels 0 .. nBins - 1)
__global__ void k_gather_levels(int64_t n, const int *idx, const int *level, uint32_t *keys, int *lvlCnt, int nBins) {
    __shared__ int h[kHistBins];
    hist_begin(h, nBins);
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        int l = level[idx[i]];
        keys[i] = (uint32_t)l;
        hist_add(h, nBins, lvlCnt, l);
    }
    hist_end(h, nBins, lvlCnt);
}

__global__ void k_inverse(int64_t n, const int *srt, int *tOf) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += stride) tOf[srt[t]] = (int)t;
}

struct DedupArgs {
    int64_t nLive;
    const int *srt;        // live AND positions in processing order
    const int *rankOf;     // per position: tentative rank (min wins)
    const int *L0, *L1;
    const int *level;
    const int *lvlCnt;     // live AND nodes per level
    const int *lvlStart;   // first processing index of each level
    const int *chunkStart; // first chunk of each level (maxLevel + 2 entries)
    int maxLevel;
    int *lvlDone;
    const int *gid;
    const DevGraph *dg;
    AndTable tab;
    int *mapEnc;  // per position: mapped literal (>= 0) or -(slot+1)
    int *kl0, *kl1;
    int *slotT;   // per processing index: table slot, -1 when folded
    int foldTrivial;
    int unique;  // key each node by its position: nothing merges
    int *counter;
    int *status;
};

constexpr int kDedupChunk = kBlock;

__device__ __forceinline__ int resolve_map(const DedupArgs &A, int u) {
    int e = __ldcg(&A.mapEnc[u]);
    if (e >= 0) return e;
    return 2 * slot_pos(__ldcg(&A.tab.slots[-e - 1].rp));
}

// chunks per level, for the level-aligned claim order of k_dedup
__global__ void k_level_chunks(int n, const int *lvlCnt, int *cc) {
    int stride = gridDim.x * blockDim.x;
    for (int l = blockIdx.x * blockDim.x + threadIdx.x; l < n; l += stride)
        cc[l] = (lvlCnt[l] + kDedupChunk - 1) / kDedupChunk;
}

// Dataflow over the processing order in chunks that never cross a level.
// A chunk of level L needs its fanins' levels (< L) hashed: one thread waits
// for the highest of them, since a level completes only after the level
// below it has (every node of level L has a fanin on level L - 1).  The
// chunk then maps, folds and hashes its nodes and adds its size to its
// level's completion counter with one atomic.
__global__ void __launch_bounds__(kDedupChunk) k_dedup(DedupArgs A) {
    __shared__ int s_begin, s_end, s_level, s_need, s_ok;
    while (true) {
        if (threadIdx.x == 0) {
            const int c = atomicAdd(A.counter, 1);
            if (c < A.chunkStart[A.maxLevel + 1]) {
                int lo = 0, hi = A.maxLevel;
                while (lo < hi) {  // last level whose first chunk is <= c
                    int mid = (lo + hi + 1) >> 1;
                    if (A.chunkStart[mid] <= c)
                        lo = mid;
                    else
                        hi = mid - 1;
                }
                const int b = A.lvlStart[lo] + (c - A.chunkStart[lo]) * kDedupChunk;
                const int e = A.lvlStart[lo] + A.lvlCnt[lo];
                s_begin = b;
                s_end = b + kDedupChunk < e ? b + kDedupChunk : e;
                s_level = lo;
            } else {
                s_begin = -1;
            }
            s_need = -1;
        }
        __syncthreads();
        const int begin = s_begin, end = s_end, lv = s_level;
        if (begin < 0) break;
        const int t = begin + (int)threadIdx.x;
        const bool valid = t < end;
        int v = 0, lits[2] = {0, 0};
        if (valid) {
            v = A.srt[t];
            lits[0] = A.L0[v];
            lits[1] = A.L1[v];
            int need = -1;
            for (int k = 0; k < 2; k++) {
                const int u = lits[k] >> 1;
                if (A.L0[u] >= 0) need = max(need, A.level[u]);
            }
            if (need >= 0) atomicMax(&s_need, need);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            const int need = s_need;
            s_ok = need < 0 ? 1 : (wait_ge(&A.lvlDone[need], A.lvlCnt[need], A.status) ? 1 : 0);
        }
        __syncthreads();
        if (valid && s_ok) {
            for (int k = 0; k < 2; k++) {
                const int u = lits[k] >> 1;
                if (A.L0[u] < 0) continue;  // PI or constant keeps its literal
                lits[k] = resolve_map(A, u) ^ (lits[k] & 1);
            }
            int l0 = lits[0], l1 = lits[1];
            if (l0 > l1) {
                int x = l0;
                l0 = l1;
                l1 = x;
            }
            const int T = 2 * A.dg[A.gid[v]].cpos;  // AIGMan: constant TRUE
            const int F = T + 1;
            int triv = -1;
            if (A.foldTrivial) {
                if (l0 == l1)
                    triv = l0;
                else if (l0 == (l1 ^ 1))
                    triv = F;
                else if (l0 == T)
                    triv = l1;
                else if (l1 == T)
                    triv = l0;
                else if (l0 == F || l1 == F)
                    triv = F;
            }
            if (triv >= 0) {
                A.mapEnc[v] = triv;
                A.slotT[t] = -1;
            } else {
                // literals are non-negative, so a key with the top bit set
                // is never a real one
                const unsigned long long key = A.unique ? (1ull << 63) | (unsigned long long)(uint32_t)v
                                                        : ((unsigned long long)(uint32_t)l0 << 32) | (uint32_t)l1;
                int slot = table_insert(A.tab, key, A.rankOf[v], v, A.status);
                A.kl0[t] = l0;
                A.kl1[t] = l1;
                A.mapEnc[v] = slot >= 0 ? -(slot + 1) : 0;
                A.slotT[t] = slot;
            }
        }
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(&A.lvlDone[lv], end - begin);
        }
    }
}

// ------------------------------------------------- deduplication in rounds
// The mapping k_dedup computes is the unique fixed point of one parallel
// step: a node's key is its fanins' mapped literals (folded when trivial),
// and it maps to the position of the lowest-ranked live node with the same
// key.  (By induction over the levels: a node's key reads only lower levels,
// so any fixed point equals the level-by-level result.)  Starting from the
// identity, the first round keys and maps every node; a later round keys only
// the nodes with a fanin whose mapping changed, and maps again only the nodes
// of slots that received a key.  No thread waits on another, so a deep,
// narrow graph costs a few launches instead of one wait latency per level.
//
// The mappings are read and written in place, so that of two nodes that map
// alike one may move a round before the other, and keys that a node had
// earlier stay in the table.  Neither does harm.  Every mapping on the way is
// sound: what it makes equal is equal in the fixed point (nodes with equal
// keys under a sound mapping are).  So a node that was ever inserted with a
// key of the fixed point, whose literals are final ones, has that key in the
// end.  Every change is seen by the node's readers a round later, so in a round
// without any, all nodes are keyed by the mapping as it stands; by induction
// over the levels it is the fixed point: a node's fanins map right, so its key
// is final, its slot holds just the nodes of that key, and it maps to the
// lowest.
//
// A round over all nodes moves their keys and table sectors (9.5M nodes: 1.1
// ms, and merges cascade for 15 rounds on a 256-graph batch); a later round
// reads their fanins and two bits each (0.15 ms).  That batch's
// deduplication: 19.9 -> 6.6 ms; 2,000 graphs of up to 2,000 ANDs (14
// rounds): 2.7 -> 1.75 ms.
struct RoundArgs {
    int64_t nLive, M;
    const int *srt, *tOf, *rankOf;
    const uint8_t *liveFlag;
    const int *L0, *L1;
    const int *gid;
    const DevGraph *dg;
    AndTable tab;
    int *cur;    // per position: the literal an AND node maps to
    int *slotT;  // per processing index: table slot, -1 when folded
    int *mapEnc, *kl0, *kl1;
    int foldTrivial, unique;
    const uint32_t *chIn;  // per position: mapping changed in the round before
    uint32_t *chOut;       //   in this round
    uint32_t *slotBits;    // per slot: received a key in this round
    const int *prev;       // whether the round before changed anything (null: first round)
    int *changed;
    int *inserted;         // keys inserted by later rounds, at most `room`
    int room;
    int *full;             // a later round ran out of room: start again from all nodes
    int *status;
};

__device__ __forceinline__ bool bit_at(const uint32_t *b, int i) { return (b[i >> 5] >> (i & 31)) & 1u; }
__device__ __forceinline__ void set_bit(uint32_t *b, int i) { atomicOr(&b[i >> 5], 1u << (i & 31)); }

__global__ void k_round_init(int64_t n, const int *srt, int *cur) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += stride) {
        const int v = srt[t];
        cur[v] = 2 * v;
    }
}

__device__ __forceinline__ void round_map(const RoundArgs &A, int v, int lit) {
    if (A.cur[v] == lit) return;
    A.cur[v] = lit;
    set_bit(A.chOut, v);
    *A.changed = 1;
}

// Node v's key from the current mappings, folded as k_dedup does: returns the
// literal it folds to, or -1 with the key's literals in l0 <= l1.
__device__ __forceinline__ int round_key(const RoundArgs &A, int v, int &l0, int &l1) {
    l0 = A.L0[v], l1 = A.L1[v];
    if (A.L0[l0 >> 1] >= 0) l0 = A.cur[l0 >> 1] ^ (l0 & 1);
    if (A.L0[l1 >> 1] >= 0) l1 = A.cur[l1 >> 1] ^ (l1 & 1);
    if (l0 > l1) {
        const int x = l0;
        l0 = l1;
        l1 = x;
    }
    if (!A.foldTrivial) return -1;
    const int T = 2 * A.dg[A.gid[v]].cpos;  // AIGMan: constant TRUE
    const int F = T + 1;
    if (l0 == l1) return l0;
    if (l0 == (l1 ^ 1)) return F;
    if (l0 == T) return l1;
    if (l1 == T) return l0;
    if (l0 == F || l1 == F) return F;
    return -1;
}

__device__ __forceinline__ int round_insert(const RoundArgs &A, int v, int t, int l0, int l1) {
    const unsigned long long key = A.unique ? (1ull << 63) | (unsigned long long)(uint32_t)v
                                            : ((unsigned long long)(uint32_t)l0 << 32) | (uint32_t)l1;
    const int slot = table_insert(A.tab, key, A.rankOf[v], v, A.status);
    A.kl0[t] = l0;
    A.kl1[t] = l1;
    A.mapEnc[v] = slot >= 0 ? -(slot + 1) : 0;
    A.slotT[t] = slot;
    return slot;
}

// first round: every node's key
__global__ void k_round_insert(RoundArgs A) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < A.nLive; t += stride) {
        const int v = A.srt[t];
        int l0, l1;
        const int triv = round_key(A, v, l0, l1);
        if (triv >= 0) {
            A.mapEnc[v] = triv;
            A.slotT[t] = -1;
            round_map(A, v, triv);
        } else {
            round_insert(A, v, (int)t, l0, l1);
        }
    }
}

// first round: every key's lowest rank is known, and the inserted nodes map
// to its position
__global__ void k_round_resolve(RoundArgs A) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < A.nLive; t += stride) {
        const int slot = A.slotT[t];
        if (slot >= 0) round_map(A, A.srt[t], 2 * slot_pos(A.tab.slots[slot].rp));
    }
}

// later round: new keys of the nodes with a fanin that maps elsewhere now
__global__ void k_round_rekey(RoundArgs A) {
    if (*A.prev == 0) return;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < A.M; p += stride) {
        const int v = (int)p, a = A.L0[v];
        if (a < 0) continue;
        const int b = A.L1[v];
        if (!bit_at(A.chIn, a >> 1) && !bit_at(A.chIn, b >> 1)) continue;
        if (!A.liveFlag[v]) continue;
        const int t = A.tOf[v];
        int l0, l1;
        const int triv = round_key(A, v, l0, l1);
        if (triv >= 0) {
            A.mapEnc[v] = triv;
            A.slotT[t] = -1;
            round_map(A, v, triv);
        } else if (A.slotT[t] < 0 || A.kl0[t] != l0 || A.kl1[t] != l1) {
            const unsigned m = __activemask();
            const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
            int at = 0;
            if (lane == lead) at = atomicAdd(A.inserted, __popc(m));
            if (__shfl_sync(m, at, lead) + __popc(m) > A.room) {
                *A.full = 1;
                continue;
            }
            const int slot = round_insert(A, v, t, l0, l1);
            if (slot >= 0) set_bit(A.slotBits, slot);
        }
    }
}

// later round: the nodes of the slots that received a key
__global__ void k_round_remap(RoundArgs A) {
    if (*A.prev == 0) return;
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < A.nLive; t += stride) {
        const int slot = A.slotT[t];
        if (slot >= 0 && bit_at(A.slotBits, slot)) round_map(A, A.srt[t], 2 * slot_pos(A.tab.slots[slot].rp));
    }
}

// A node wins when its key's lowest rank is its own: its rank is its
// processing index, or (id order) rankOf of its position.
__global__ void k_winner_flags(int64_t n, const int *srt, const int *rankOf, bool idOrder, const int *slotT,
                               const AndSlot *slots, uint8_t *flags) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += stride) {
        const int slot = slotT[t];
        const int rank = idOrder ? rankOf[srt[t]] : (int)t;
        flags[t] = (slot >= 0 && slot_rank(slots[slot].rp) == rank) ? 1 : 0;
    }
}

__global__ void k_gather_rank(int64_t n, const int *wl, const int *srt, const int *rankOf, uint32_t *keys) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        keys[i] = (uint32_t)rankOf[srt[wl[i]]];
}

// Winners of each graph in output order: key = gid, stable.
__global__ void k_winner_keys(int64_t n, const int *wl, const int *srt, const int *gid, uint32_t *keys, int *cntG) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        int g = gid[srt[wl[i]]];
        keys[i] = (uint32_t)g;
        agg_add(cntG, g, 1);
    }
}

__global__ void k_winner_local(int64_t n, const int *wlByG, const int *srt, const int *gid, const int *gStart,
                               const DevGraph *dg, int *newLocalT) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        int t = wlByG[i];
        int g = gid[srt[t]];
        newLocalT[t] = dg[g].nPIs + 1 + (int)(i - (gStart ? gStart[g] : 0));
    }
}

struct OutArgs {
    const int *srt, *tOf, *gid, *lidIn, *L0, *kl0, *kl1, *newLocalT, *mapEnc;
    const AndSlot *slots;
    const int *po;
    const DevGraph *dgNew;
    int *F0, *F1, *PO;
    int64_t nPO, M;
};

__device__ __forceinline__ int local_lit(const OutArgs &A, int lit) {
    int u = lit >> 1;
    if (A.L0[u] < 0) return 2 * A.lidIn[u] + (lit & 1);
    return 2 * A.newLocalT[A.tOf[u]] + (lit & 1);
}

__global__ void k_strash_out(int64_t nW, const int *wl, OutArgs A) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nW; i += stride) {
        int t = wl[i];
        int v = A.srt[t];
        int g = A.gid[v];
        int p = A.dgNew[g].base + A.newLocalT[t];
        // the reference forms keys over the final numbering, so the
        // smaller literal comes first there
        int a = local_lit(A, A.kl0[t]), b = local_lit(A, A.kl1[t]);
        A.F0[p] = a < b ? a : b;
        A.F1[p] = a < b ? b : a;
    }
    // the constants and PIs
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < A.M; v += stride) {
        if (A.L0[v] >= 0) continue;
        const int p = A.dgNew[A.gid[v]].base + A.lidIn[v];
        A.F0[p] = A.F1[p] = -1;
    }
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < A.nPO; k += stride) {
        int lit = A.po[k];
        int u = lit >> 1;
        int m = lit;
        if (A.L0[u] >= 0) {
            int e = A.mapEnc[u];
            int base = e >= 0 ? e : 2 * slot_pos(A.slots[-e - 1].rp);
            m = base ^ (lit & 1);
        }
        A.PO[k] = local_lit(A, m);
    }
}

}  // namespace

int Engine::strash_core(Batch &b, int64_t M, const int *L0, const int *L1, const int *gidA, const int *lidIn,
                        const int *po, bool idOrder, bool removeDangling, bool foldTrivial, bool topo,
                        bool unique, const int *procInv, const int *procPos) {
    const int G = b.G;
    const int64_t nPO = b.nPO;
    cudaStream_t s = s_;
    int *cnt = ar_.get<int>(M + 1);
    uint8_t *dead = ar_.get<uint8_t>(M + 1);
    uint8_t *flags = ar_.get<uint8_t>(M + 1);
    uint8_t *liveFlag = ar_.get<uint8_t>(M + 1);
    int *items = ar_.get<int>(M + 1);
    int *level = ar_.get<int>(M + 1);
    int *pending = ar_.get<int>(M + 1);
    int *off = ar_.get<int>(M + 2);
    int *graphLevels = ar_.get<int>(G + 1);
    if (!cnt || !dead || !flags || !liveFlag || !items || !level || !pending || !off || !graphLevels)
        return fail(CULS_E_OOM, "strash: scratch arena exhausted");
    int *qc = counters_;  // [0]=head [1]=tail [2]=done [3]=count [4]=maxLevel [5]=counter
    const unsigned gridM = grid_1d(std::max<int64_t>(M, nPO), kBlock, sms_ * 16);
    const unsigned gridQ = flow_blocks(b.flow_width(), kBlock, (unsigned)(sms_ * 8), sms_);

    // 1. liveness
    check(cudaMemsetAsync(dead, 0, (size_t)M + 1, s), "memset");
    if (removeDangling) {
        check(cudaMemsetAsync(cnt, 0, sizeof(int) * (M + 1), s), "memset");
        k_fanout_count<<<gridM, kBlock, 0, s>>>(M, L0, L1, po, nPO, cnt);
        k_dead_seed_flags<<<gridM, kBlock, 0, s>>>(M, L0, cnt, flags);
        check(fill_i32(items, -1, M + 1, s), "fill");
        check(cudaMemsetAsync(qc, 0, sizeof(int) * 8, s), "memset");
        if (int e = check(compact_flags(flags, M, items, qc + 1, ar_, s), "compact")) return e;
        k_dead_queue<<<gridQ, kBlock, 0, s>>>(WorkQueue{items, qc + 0, qc + 1, qc + 2, (int)(M + 1)}, L0, L1, cnt,
                                              dead, status_);
        launches_ += 4;
    }
    // 2. levels of live AND nodes
    int *liveIdx = nullptr;
    if (topo) {
        liveIdx = ar_.get<int>(M + 1);
        int *done = pending;  // reuse
        if (!liveIdx) return fail(CULS_E_OOM, "strash: scratch arena exhausted");
        ExecCtx X = ctx();
        const bool inBlock = G == 1 && M <= kLevelsBlockMax;
        ChunkSched sched;
        int rc;
        if (!inBlock && (rc = build_chunk_sched(X, b, kBlock, sched))) return rc;
        check(cudaMemsetAsync(qc, 0, sizeof(int) * 8, s), "memset");
        check(cudaMemsetAsync(graphLevels, 0, sizeof(int) * (G + 1), s), "memset");
        check(cudaMemsetAsync(level, 0, sizeof(int) * (M + 1), s), "memset");
        k_live_flags<<<gridM, kBlock, 0, s>>>(M, L0, dead, liveFlag, done);
        if (int e = check(compact_flags(liveFlag, M, liveIdx, qc + 3, ar_, s), "compact")) return e;  // live list and count
        if (prof_) this->mark(kMkLevelK0);
        if (inBlock) {
            LevelsArgs A;
            A.n = M, A.a0 = L0, A.a1 = L1, A.level = level, A.counted = liveFlag;
            A.depth0 = qc + 4, A.depth1 = graphLevels, A.unsettled = qc + 6, A.status = status_;
            if ((rc = check(levels_block(A, s), "levels"))) return rc;
        } else {
            k_st_levelize<<<gridQ, kBlock, 0, s>>>(sched, L0, L1, liveFlag, gidA, level, done, graphLevels, qc + 5,
                                                   qc + 4, status_);
        }
        if (prof_) this->mark(kMkLevelK1);
        launches_ += 2;
    } else {
    // in-order passes over procInv; the worklist below is the fallback if a
    // pass stops making progress (a cycle) or a wait times out, and runs
    // alone when CULS_DEDUP_WORKLIST is set (the tests compare the two)
    bool leveled = false;
    if (procInv && !getenv("CULS_DEDUP_WORKLIST")) {
        liveIdx = ar_.get<int>(M + 1);
        if (!liveIdx) return fail(CULS_E_OOM, "strash: scratch arena exhausted");
        int *done = pending;
        int *lists[2] = {cnt, off};  // free until the levels are known
        int *idx = items;
        check(cudaMemsetAsync(qc, 0, sizeof(int) * 8, s), "memset");
        // qc[7] is these passes' own status word; qc[8] its spin bound
        check(cudaMemcpyAsync(qc + 8, status_ + 1, sizeof(int), cudaMemcpyDeviceToDevice, s), "copy");
        check(cudaMemsetAsync(graphLevels, 0, sizeof(int) * (G + 1), s), "memset");
        check(cudaMemsetAsync(level, 0, sizeof(int) * (M + 1), s), "memset");
        k_live_flags<<<gridM, kBlock, 0, s>>>(M, L0, dead, liveFlag, done);
        if (int e = check(compact_flags(liveFlag, M, liveIdx, qc + 3, ar_, s), "compact")) return e;  // live list and count
        launches_ += 1;
        if (prof_) this->mark(kMkLevelK0);
        const int *list = procInv;
        int64_t n = M;
        if (G == 1 && M <= kLevelsBlockMax) {
            int *a0 = cnt, *a1 = off;
            k_order_fanins<<<gridM, kBlock, 0, s>>>(M, procInv, procPos, L0, L1, liveFlag, a0, a1);
            LevelsArgs A;
            A.n = M, A.a0 = a0, A.a1 = a1, A.posOf = procInv, A.level = level;
            A.depth0 = qc + 4, A.depth1 = graphLevels, A.unsettled = qc + 6, A.status = qc + 7;
            if (int e = check(levels_block(A, s), "levels")) return e;
            launches_ += 2;
            if (int e = fetch("strash levels")) return e;
            leveled = hostSmall_[6] == 0 && hostSmall_[7] == 0;
        } else
        for (int pass = 0; pass < 64; pass++) {
            check(cudaMemsetAsync(qc + 5, 0, sizeof(int), s), "memset");
            k_order_levelize<<<gridQ, kBlock, 0, s>>>(n, list, procPos, L0, L1, liveFlag, gidA, level, done,
                                                      graphLevels, qc + 5, qc + 4, qc + 7);
            k_unresolved_flags<<<grid_1d(n, kBlock, sms_ * 16), kBlock, 0, s>>>(n, list, done, flags);
            launches_ += 2;
            if (int e = check(compact_flags(flags, n, idx, qc + 6, ar_, s), "compact")) return e;
            if (int e = fetch("strash levels")) return e;
            const int64_t nu = hostSmall_[6];
            if (hostSmall_[7] != 0) break;  // a wait timed out
            if (nu == 0) {
                leveled = true;
                break;
            }
            if (pass > 0 && nu == n) break;  // no progress
            int *next = lists[pass & 1];
            k_unresolved_next<<<grid_1d(nu, kBlock, sms_ * 16), kBlock, 0, s>>>(nu, idx, list, next, done);
            launches_ += 1;
            list = next;
            n = nu;
        }
        if (leveled && prof_) this->mark(kMkLevelK1);
    }
    if (!leveled) {
    check(cudaMemsetAsync(off, 0, sizeof(int) * (M + 2), s), "memset");
    k_live_degrees<<<gridM, kBlock, 0, s>>>(M, L0, L1, dead, level, off, liveFlag, flags);
    if (int e = check(scan_exclusive(off, off, M + 1, nullptr, ar_, s), "scan")) return e;
    int *cursor = cnt;  // reuse
    check(cudaMemcpyAsync(cursor, off, sizeof(int) * (M + 1), cudaMemcpyDeviceToDevice, s), "copy");
    // number of live edges = off[M]
    check(cudaMemcpyAsync(hostSmall_, off + M, sizeof(int), cudaMemcpyDeviceToHost, s), "d2h");
    if (int e = sync()) return e;
    int64_t nEdges = hostSmall_[0];
    int *adj = ar_.get<int>(nEdges + 1);
    if (!adj) return fail(CULS_E_OOM, "strash: scratch arena exhausted");
    k_csr_fill<<<gridM, kBlock, 0, s>>>(M, L0, L1, liveFlag, cursor, adj);
    liveIdx = ar_.get<int>(M + 1);
    int *ring = ar_.get<int>(8);
    if (!liveIdx || !ring) return fail(CULS_E_OOM, "strash: scratch arena exhausted");
    check(cudaMemsetAsync(qc, 0, sizeof(int) * 8, s), "memset");
    check(cudaMemsetAsync(ring, 0, sizeof(int) * 8, s), "memset");
    check(cudaMemsetAsync(graphLevels, 0, sizeof(int) * (G + 1), s), "memset");
    if (int e = check(compact_flags(flags, M, items, ring + 1, ar_, s), "compact")) return e;     // level 1: the seeds
    if (int e = check(compact_flags(liveFlag, M, liveIdx, qc + 3, ar_, s), "compact")) return e;  // live list and count
    launches_ += 2;
    if (prof_) this->mark(kMkLevelK0);
    // levels in launches of 64, until a level comes out empty; the ring
    // then holds the number of nodes given a level (all live ones unless
    // there is a cycle)
    int L = 1;
    while (true) {
        for (int t = 0; t < 64; t++, L++)
            k_level_step<<<gridQ, kBlock, 0, s>>>(L, items, ring, off, adj, L0, L1, level, gidA, graphLevels, qc + 4);
        launches_ += 64;
        check(cudaMemcpyAsync(hostSmall_, ring, sizeof(int) * 6, cudaMemcpyDeviceToHost, s), "d2h");
        if (int e = sync()) return e;
        if (hostSmall_[L % 3] == 0) break;
    }
    check(cudaMemcpyAsync(qc + 1, ring + 3 + L % 3, sizeof(int), cudaMemcpyDeviceToDevice, s), "copy");
    if (prof_) this->mark(kMkLevelK1);
    if (int e = fetch("strash levels")) return e;
    if (hostSmall_[1] != hostSmall_[3]) return fail(CULS_E_INVALID, "strash: the AIG has a cycle");
    }
    }
    // 3. processing order (level, position) and tentative ranks
    if (topo) {
        if (int e = fetch("strash levels")) return e;
        if (hostSmall_[6]) return fail(CULS_E_INVALID, "strash: fanins do not precede their node");
    }
    const int64_t nLive = hostSmall_[3];
    const int maxLevel = hostSmall_[4];
    int *srt = ar_.get<int>(nLive + 1);
    uint32_t *keys = ar_.get<uint32_t>(nLive + 1);
    uint32_t *keys2 = ar_.get<uint32_t>(nLive + 1);
    int *vals2 = ar_.get<int>(nLive + 1);
    int *lvlCnt = ar_.get<int>(maxLevel + 2);
    int *lvlDone = ar_.get<int>(maxLevel + 2);
    int *lvlStart = ar_.get<int>(maxLevel + 2);
    int *chunkCnt = ar_.get<int>(maxLevel + 2);
    int *chunkStart = ar_.get<int>(maxLevel + 2);
    int *tOf = pending;  // reuse
    int *rankOf = off;   // reuse (only needs M entries)
    if (!srt || !keys || !keys2 || !vals2 || !lvlCnt || !lvlDone || !lvlStart || !chunkCnt || !chunkStart)
        return fail(CULS_E_OOM, "strash: arena exhausted");
    check(cudaMemsetAsync(lvlCnt, 0, sizeof(int) * (maxLevel + 2), s), "memset");
    if (nLive > 0) {
        unsigned gl = grid_1d(nLive, kBlock, sms_ * 16);
        k_gather_levels<<<gl, kBlock, 0, s>>>(nLive, liveIdx, level, keys, lvlCnt, maxLevel + 1);
        int bits = 1;
        while ((1ll << bits) <= maxLevel) bits++;
        check(cudaMemcpyAsync(vals2, liveIdx, sizeof(int) * nLive, cudaMemcpyDeviceToDevice, s), "copy");
        if (int e = check(radix_sort_pairs(keys, vals2, keys2, srt, nLive, bits, ar_, s), "sort")) return e;
        k_inverse<<<gl, kBlock, 0, s>>>(nLive, srt, tOf);
        // tentative rank: processing order, or id order for the CPU variants
        k_inverse<<<gl, kBlock, 0, s>>>(nLive, idOrder ? liveIdx : srt, rankOf);
        launches_ += 3;
    }
    // 4. hash: fixed-point rounds or the level dataflow (below)
    uint32_t cap = 1024;
    while (cap < (uint32_t)std::min<int64_t>(nLive * 2, 1ll << 31)) cap <<= 1;
    // CULS_STRASH_TABLE_CAP lowers the capacity (rounded up to a power of
    // two): the tests use it to make the bounded probes run out and check
    // that the call reports CULS_E_PROBE and leaves the graph as it was
    if (const char *env = getenv("CULS_STRASH_TABLE_CAP")) {
        const long long want = atoll(env);
        if (want >= 1) {
            uint32_t c = 1;
            while ((long long)c < want && c < (1u << 31)) c <<= 1;
            cap = std::min(cap, c);
        }
    }
    AndSlot *ts = ar_.get<AndSlot>(cap);
    int *mapEnc = ar_.get<int>(M + 1);
    int *kl0 = ar_.get<int>(nLive + 1), *kl1 = ar_.get<int>(nLive + 1);
    uint8_t *wflags = ar_.get<uint8_t>(nLive + 1);
    int *wl = ar_.get<int>(nLive + 1);
    if (!ts || !mapEnc || !kl0 || !kl1 || !wflags || !wl) return fail(CULS_E_OOM, "strash: arena exhausted");
    // Rounds (k_round_*) for batches of up to 16M live nodes, where a full
    // pass and a few light ones cost less than one wait latency per level
    // (the 10M-AND single graph: each strash 22 -> 6 ms); the level dataflow
    // (k_dedup) for larger ones, whose rounds each move gigabytes and whose
    // merges can cascade for many rounds, and whenever the rounds do not
    // settle within kMaxHashRounds.  CULS_DEDUP_MODE=levels|rounds forces either
    // (the tests run both on the same graphs).
    constexpr int64_t kRoundsMaxLive = 16ll << 20;
    bool useRounds = nLive > 0 && nLive <= kRoundsMaxLive;
    if (const char *env = getenv("CULS_DEDUP_MODE")) {
        if (!strcmp(env, "levels")) useRounds = false;
        if (!strcmp(env, "rounds")) useRounds = nLive > 0;
    }
    bool settled = false;
    hashRounds_ = 0;
    int *slotT = ar_.get<int>(nLive + 1);
    if (!slotT) return fail(CULS_E_OOM, "strash: arena exhausted");
    if (useRounds) {
        int *cur = ar_.get<int>(M + 1), *flag = counters_ + kCtRound;
        const size_t posWords = (size_t)M / 32 + 1, slotWords = (size_t)cap / 32 + 1;
        uint32_t *ch[2] = {ar_.get<uint32_t>(posWords), ar_.get<uint32_t>(posWords)};
        uint32_t *slotBits = ar_.get<uint32_t>(slotWords);
        if (!cur || !ch[0] || !ch[1] || !slotBits) return fail(CULS_E_OOM, "strash: arena exhausted");
        const unsigned gl = grid_1d(nLive, kBlock, sms_ * 16);
        if (prof_) this->mark(kMkDedupK0);
        k_round_init<<<gl, kBlock, 0, s>>>(nLive, srt, cur);
        launches_ += 1;
        // later rounds' keys come on top of every node's first: a quarter of
        // the table, or what a lowered capacity leaves
        const int room = (int)std::min<int64_t>(cap / 4, std::max<int64_t>((int64_t)cap - nLive, 0));
        RoundArgs R{nLive, M,   srt,    tOf, rankOf, liveFlag, L0, L1, gidA, b.dg, AndTable{ts, cap - 1}, cur, slotT,
                    mapEnc, kl0, kl1,   foldTrivial ? 1 : 0, unique ? 1 : 0, nullptr, nullptr, slotBits, nullptr, nullptr,
                    counters_ + kCtInserted, room, counters_ + kCtFull, status_};
        check(cudaMemsetAsync(flag, 0, sizeof(int) * kMaxHashRounds, s), "memset");
        bool all = true;  // the next round takes all nodes
        for (int r = 0; r < kMaxHashRounds && !settled;) {
            // per host check three rounds, or one over all nodes where
            // nothing is expected to merge (a round that follows one without
            // a change does nothing)
            const int first = r, last = std::min(all && topo ? r + 1 : r + 3, kMaxHashRounds);
            for (; r < last; r++) {
                R.chIn = ch[(r + 1) & 1], R.chOut = ch[r & 1];
                R.prev = r > 0 ? flag + r - 1 : nullptr;
                R.changed = flag + r;
                check(cudaMemsetAsync(R.chOut, 0, sizeof(uint32_t) * posWords, s), "memset");
                if (all) {
                    check(and_table_clear(ts, cap, s), "fill");
                    check(cudaMemsetAsync(R.inserted, 0, sizeof(int) * 2, s), "memset");
                    k_round_insert<<<gl, kBlock, 0, s>>>(R);
                    k_round_resolve<<<gl, kBlock, 0, s>>>(R);
                    all = false;
                } else {
                    check(cudaMemsetAsync(slotBits, 0, sizeof(uint32_t) * slotWords, s), "memset");
                    k_round_rekey<<<gridM, kBlock, 0, s>>>(R);
                    k_round_remap<<<gl, kBlock, 0, s>>>(R);
                }
                launches_ += 2;
            }
            if (int e = fetch("strash hashing")) return e;
            all = hostSmall_[kCtFull] != 0;
            for (int k = first; k < last && !settled && !all; k++)
                if (hostSmall_[kCtRound + k] == 0) {
                    settled = true;
                    hashRounds_ = k + 1;
                }
        }
        if (prof_) this->mark(kMkDedupK1);
    }
    if (nLive > 0 && !settled) {
        // level-aligned chunks for the hashing dataflow
        check(cudaMemsetAsync(lvlDone, 0, sizeof(int) * (maxLevel + 2), s), "memset");
        check(cudaMemsetAsync(qc + 5, 0, sizeof(int), s), "memset");
        k_level_chunks<<<grid_1d(maxLevel + 1, kBlock, sms_ * 16), kBlock, 0, s>>>(maxLevel + 1, lvlCnt, chunkCnt);
        if (int e = check(scan_exclusive(lvlCnt, lvlStart, maxLevel + 1, nullptr, ar_, s), "scan")) return e;
        if (int e = check(scan_exclusive(chunkCnt, chunkStart, maxLevel + 1, chunkStart + maxLevel + 1, ar_, s), "scan")) return e;
        launches_ += 1;
        check(and_table_clear(ts, cap, s), "fill");
        DedupArgs A{nLive,      srt,      rankOf,
                    L0,         L1,       level,   lvlCnt,
                    lvlStart,   chunkStart, maxLevel, lvlDone,
                    gidA,       b.dg,     AndTable{ts, cap - 1}, mapEnc,
                    kl0,        kl1,      slotT,   foldTrivial ? 1 : 0, unique ? 1 : 0,
                    qc + 5,     status_};
        if (prof_) this->mark(kMkDedupK0);
        k_dedup<<<gridQ, kBlock, 0, s>>>(A);
        if (prof_) this->mark(kMkDedupK1);
        launches_ += 1;
    }
    if (nLive > 0) {
        k_winner_flags<<<grid_1d(nLive, kBlock, sms_ * 16), kBlock, 0, s>>>(nLive, srt, rankOf, idOrder, slotT, ts, wflags);
        launches_ += 1;
    }
    if (int e = check(compact_flags(wflags, nLive, wl, qc + 6, ar_, s), "compact")) return e;
    // In id order (CPU variants) the winners are ranked by position, not by
    // processing order: sort the winner list by rank.
    if (int e = fetch("strash hashing")) return e;
    const int64_t nW = hostSmall_[6];
    int *newLocalT = ar_.get<int>(nLive + 1);
    int *cntG = ar_.get<int>(G + 1);
    int *gStart = ar_.get<int>(G + 1);
    int *wlByG = ar_.get<int>(nW + 1);
    uint32_t *wk = ar_.get<uint32_t>(nW + 1), *wk2 = ar_.get<uint32_t>(nW + 1);
    int *wv = ar_.get<int>(nW + 1);
    if (!newLocalT || !cntG || !gStart || !wlByG || !wk || !wk2 || !wv) return fail(CULS_E_OOM, "strash: arena");
    if (idOrder && nW > 0) {
        // re-order winners by id order: key = rank (position order)
        // (ranks fit in 31 bits)
        int bits = 1;
        while ((1ll << bits) <= nLive) bits++;
        k_gather_rank<<<grid_1d(nW, kBlock, sms_ * 16), kBlock, 0, s>>>(nW, wl, srt, rankOf, wk);
        check(cudaMemcpyAsync(wv, wl, sizeof(int) * nW, cudaMemcpyDeviceToDevice, s), "copy");
        if (int e = check(radix_sort_pairs(wk, wv, wk2, wl, nW, bits, ar_, s), "sort")) return e;
        launches_ += 1;
    }
    std::vector<int> hCnt(G), hLev(G);
    if (G == 1) {
        hCnt[0] = (int)nW;
        hLev[0] = maxLevel;
        wlByG = wl;
        gStart = nullptr;
    } else {
        check(cudaMemsetAsync(cntG, 0, sizeof(int) * (G + 1), s), "memset");
        if (nW > 0) {
            unsigned gw = grid_1d(nW, kBlock, sms_ * 16);
            k_winner_keys<<<gw, kBlock, 0, s>>>(nW, wl, srt, gidA, wk, cntG);
            launches_ += 1;
            int bits = 1;
            while ((1ll << bits) < G) bits++;
            check(cudaMemcpyAsync(wv, wl, sizeof(int) * nW, cudaMemcpyDeviceToDevice, s), "copy");
            if (int e = check(radix_sort_pairs(wk, wv, wk2, wlByG, nW, bits, ar_, s), "sort")) return e;
        }
        if (int e = check(scan_exclusive(cntG, gStart, G, nullptr, ar_, s), "scan")) return e;
        check(cudaMemcpyAsync(hCnt.data(), cntG, sizeof(int) * G, cudaMemcpyDeviceToHost, s), "d2h");
        check(cudaMemcpyAsync(hLev.data(), graphLevels, sizeof(int) * G, cudaMemcpyDeviceToHost, s), "d2h");
        if (int e = sync()) return e;
    }
    // new graph table
    std::vector<DevGraph> ng = b.hg;
    int64_t base = 0;
    for (int g = 0; g < G; g++) {
        ng[g].nAnds = hCnt[g];
        // the CPU strash reports maxDelay, -1 without AND nodes
        // (src/aig/strash.cu:396,454)
        ng[g].nLevels = (idOrder && hCnt[g] == 0) ? -1 : hLev[g];
        ng[g].base = (int)base;
        base += 1 + ng[g].nPIs + hCnt[g];
    }
    int64_t nObjNew = base;
    DevGraph *dgNew = reinterpret_cast<DevGraph *>(ar_.get<char>(sizeof(DevGraph) * (G + 1)));
    if (!dgNew) return fail(CULS_E_OOM, "strash: arena");
    // the output goes to the batch's spare buffers, swapped in at the end
    if (!b.pool) b.pool = pool_;
    if (int e = check(b.reserve_spare(nObjNew + 1, nPO + 1), "cudaMalloc")) return e;
    int *F0n = b.F0s, *F1n = b.F1s, *POn = b.POs;
    check(cudaMemcpyAsync(dgNew, ng.data(), sizeof(DevGraph) * G, cudaMemcpyHostToDevice, s), "h2d");
    if (nW > 0) {
        unsigned gw = grid_1d(nW, kBlock, sms_ * 16);
        k_winner_local<<<gw, kBlock, 0, s>>>(nW, wlByG, srt, gidA, gStart, b.dg, newLocalT);
        launches_ += 1;
    }
    OutArgs O{srt, tOf, gidA, lidIn, L0, kl0, kl1, newLocalT, mapEnc, ts, po, dgNew, F0n, F1n, POn, nPO, M};
    k_strash_out<<<gridM, kBlock, 0, s>>>(nW, wl, O);
    launches_ += 1;
    check(cudaMemcpyAsync(b.dg, ng.data(), sizeof(DevGraph) * G, cudaMemcpyHostToDevice, s), "h2d");
    if (int e = fetch("strash output")) return e;
    b.swap_spare();
    b.hg = ng;
    b.nObj = nObjNew;
    ar_.reset();
    return 0;
}

namespace {

// AIGMan literals of graph-major arrays to position literals (-1 for the
// constant and PIs), and each position's graph.
__global__ void k_depth_prep(int64_t N, int G, const DevGraph *dg, const int *F0, const int *F1, int *L0, int *L1,
                             int *gid) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += stride) {
        const int g = graph_of_pos(dg, G, (int)p);
        const int base = dg[g].base;
        gid[p] = g;
        if ((int)p - base <= dg[g].nPIs) {
            L0[p] = L1[p] = -1;
        } else {
            L0[p] = F0[p] + 2 * base;
            L1[p] = F1[p] + 2 * base;
        }
    }
}

}  // namespace

// AIGMan::readFromMemory's nLevels for every graph of b (the level of its
// deepest AND node, dangling ones included), by the st levelization.
int Engine::batch_depth(Batch &b) {
    const int64_t N = b.nObj;
    const int G = b.G;
    int rc;
    if ((rc = ensure_arena((size_t)N * 24 + ((size_t)64 << 20)))) return rc;
    ar_.reset();
    int *L0 = ar_.get<int>(N + 1), *L1 = ar_.get<int>(N + 1), *gid = ar_.get<int>(N + 1), *level = ar_.get<int>(N + 1),
        *done = ar_.get<int>(N + 1), *graphLevels = ar_.get<int>(G + 1);
    uint8_t *dead = ar_.get<uint8_t>(N + 1), *live = ar_.get<uint8_t>(N + 1);
    if (!L0 || !L1 || !gid || !level || !done || !graphLevels || !dead || !live)
        return fail(CULS_E_OOM, "depth: arena exhausted");
    cudaStream_t s = s_;
    ExecCtx X = ctx();
    for (auto &g : b.hg) g.cpos = g.base;
    if ((rc = check(cudaMemcpyAsync(b.dg, b.hg.data(), sizeof(DevGraph) * G, cudaMemcpyHostToDevice, s), "h2d")))
        return rc;
    ChunkSched sched;
    if ((rc = build_chunk_sched(X, b, kBlock, sched))) return rc;
    int *qc = counters_;
    if ((rc = check(cudaMemsetAsync(qc, 0, sizeof(int) * 8, s), "memset"))) return rc;
    if ((rc = check(cudaMemsetAsync(graphLevels, 0, sizeof(int) * (G + 1), s), "memset"))) return rc;
    if ((rc = check(cudaMemsetAsync(level, 0, sizeof(int) * (N + 1), s), "memset"))) return rc;
    if ((rc = check(cudaMemsetAsync(dead, 0, (size_t)N + 1, s), "memset"))) return rc;
    k_depth_prep<<<X.grid(N), kBlock, 0, s>>>(N, G, b.dg, b.F0, b.F1, L0, L1, gid);
    k_live_flags<<<X.grid(N), kBlock, 0, s>>>(N, L0, dead, live, done);
    k_st_levelize<<<flow_blocks(b.flow_width(), kBlock, (unsigned)(sms_ * 8), sms_), kBlock, 0, s>>>(sched, L0, L1, live, gid, level, done, graphLevels, qc + 5,
                                                          qc + 4, status_);
    launches_ += 3;
    std::vector<int> hl(G);
    if ((rc = check(cudaMemcpyAsync(hl.data(), graphLevels, sizeof(int) * G, cudaMemcpyDeviceToHost, s), "d2h")))
        return rc;
    if ((rc = fetch("depth"))) return rc;
    for (int g = 0; g < G; g++) b.hg[g].nLevels = hl[g];
    rc = check(cudaMemcpyAsync(b.dg, b.hg.data(), sizeof(DevGraph) * G, cudaMemcpyHostToDevice, s), "h2d");
    ar_.reset();
    return rc ? rc : sync();
}

}  // namespace culs
