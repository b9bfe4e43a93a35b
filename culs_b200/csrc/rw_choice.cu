// Conflict-free replacement and redundancy removal: the sequential choice
// loop of rw::CPUSolver::Rewrite (CULS src/algorithms/rewrite.cu:830-921,
// rewrite.h:118-124,208-220) moved onto the GPU.
//
// Choice: one block per graph works through that graph's candidates in id
// order, a window of them at a time (k_choice).  Every thread of the window
// replays one candidate -- install, FastDelete, commit or revert, step by
// step as the reference's recursion does (its order of reference-count
// updates matters when a cone reaches a node along two paths: a node can be
// deleted twice) -- against the committed graph, with its own changes kept in
// a small overlay.  A candidate that read something which an earlier candidate
// of the window changes -- a deletion flag, a fanin, or a reference count that
// may now be zero where it was not, or the other way round -- has seen a stale
// graph; everything before the first such candidate is exactly what the
// sequential loop would have done, is committed at once, and the next window
// starts there.
//
// Redundancy removal chases buffer chains.  The reference does it in one
// sequential sweep in which a node's fanins, once rewritten, can make it
// redundant for later nodes only.  Here every node computes its chased fanins
// in parallel, judging each node it passes "as of its own id"; the sweep is
// repeated until nothing changes, which reproduces the sequential result
// because a node's outcome depends only on nodes with smaller ids.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>

#include <cooperative_groups.h>

#include "rw_work.cuh"

namespace cg = cooperative_groups;

namespace culs {

namespace {

// Nodes a candidate may touch in its overlay, and frames of its traversal
// stack.  On the 1M-AND layered graph (rw -z) candidates touch 5 nodes above
// the inputs on average and at most 53 reads of 24 traversed nodes; a
// candidate that needs more is replayed alone on the committed graph.
constexpr int kOverlay = 32;  // a multiple of 8
constexpr int kSpecFrames = 16;

// Candidates replayed one after another at a stretch, at most (see k_choice).
constexpr int kMaxAlone = 64;

struct ChoiceArgs {
    int64_t nL0;  // W positions [0, nL0) are constants and PIs
    const DevGraph *dg;
    int4 *rec;                // per node {L0, L1, ref, del}
    int4 *mark;               // per node, by the window's candidates: lowest place that changes its flag, its count
                              // (INT_MAX: none), what is taken from its count in all, lowest place that changes its fanins
    const int4 *recA, *recB;  // per candidate in graph order: {c, q, rep, -}, leaves
    const int *gStart, *gCount;  // a graph's candidates (several graphs)
    int n;                       // all candidates
    int useZeros;
    int serial;  // replay every candidate alone
    int4 *stack;
    int stackCap;
    int *choice;
    unsigned long long *stats;  // replaced, pos, zero, reverted, compromised, selfRef, expected
    int *status;
};

// Handles.  A node above the constant and the PIs is changed through its
// handle; the constant and the PIs have none (-1): their counts
// never decide anything (FastDelete does not enter them), they are never
// deleted, and the choice's caller does not read them, so nothing is kept
// for them.

// The committed graph, changed in place by one thread between two barriers of
// its block or cluster (so its loads may come from L1); a node's handle is its
// position.
struct GraphMem {
    int4 *rec;
    int64_t nL0;
    __device__ __forceinline__ int4 ld(int x) const { return rec[x]; }
    __device__ __forceinline__ int append(int x, const int4 &) const { return x >= nL0 ? x : -1; }
    __device__ __forceinline__ void slots(int x0, const int4 &, int x1, const int4 &, int &k0, int &k1) const {
        k0 = x0 >= nL0 ? x0 : -1;
        k1 = x1 >= nL0 ? x1 : -1;
    }
    __device__ __forceinline__ int del(int k) const { return k >= 0 ? rec[k].w : 0; }
    __device__ __forceinline__ int ref(int k, int base) const { return k >= 0 ? rec[k].z : base; }
    __device__ __forceinline__ void add(int k, int d) {
        if (k >= 0) rec[k].z += d;
    }
    __device__ __forceinline__ void set_del(int k, int v) { rec[k].w = v; }
    __device__ __forceinline__ void use_del(int) {}
    __device__ __forceinline__ void use_fanins(int) {}
    __device__ __forceinline__ void decide(int, int) {}
    __device__ __forceinline__ void set_fanins(int k, int a, int b) {
        rec[k].x = a;
        rec[k].y = b;
    }
    __device__ __forceinline__ bool failed() const { return false; }
};

// The committed graph under one candidate's changes; a node's handle is its
// entry in the thread's overlay.  Entry k: node id and {deleted before: bit
// 0, deleted now: bit 1, fanins rewritten: bit 2, flag mattered: bit 3, a count
// that was zero or below mattered: bit 4, fanins mattered: bit 5, lowest
// positive count that mattered: bits 6-15 (kNoLow: none), change of ref: bits
// 16-31}.  The ids lie four to a 16-byte word, words and states thread-minor
// in shared memory.
constexpr int kNoLow = 1023;
// OneSm: all threads that change the graph are on one SM, whose L1 may hold it.
template <bool OneSm>
struct OverlayMem {
    const int4 *rec;
    int64_t nL0;
    int4 *ids;
    int *sts;
    int stride;
    int n;
    bool full;
    __device__ __forceinline__ int4 ld(int x) const { return OneSm ? rec[x] : __ldcg(rec + x); }
    __device__ __forceinline__ int id(int k) const { return reinterpret_cast<const int *>(ids + (k >> 2) * stride)[k & 3]; }
    // new entry of node x with record r; x has none
    __device__ __forceinline__ int append(int x, const int4 &r) {
        if (x < nL0) return -1;
        if (n == kOverlay) {
            full = true;
            return 0;  // the candidate is abandoned, so any entry will do
        }
        reinterpret_cast<int *>(ids + (n >> 2) * stride)[n & 3] = x;
        sts[n * stride] = (r.w ? 3 : 0) | (kNoLow << 6);
        return n++;
    }
    // the entries of x0 and x1, made when absent (places beyond n hold
    // leftovers, which are not entries)
    __device__ __forceinline__ void slots(int x0, const int4 &r0, int x1, const int4 &r1, int &k0, int &k1) {
        k0 = k1 = -1;
        for (int k = 0; k < n; k += 4) {
            const int4 v = ids[(k >> 2) * stride];
            const int left = n - k;
            if (v.x == x0) k0 = k;
            if (v.x == x1) k1 = k;
            if (v.y == x0 && left > 1) k0 = k + 1;
            if (v.y == x1 && left > 1) k1 = k + 1;
            if (v.z == x0 && left > 2) k0 = k + 2;
            if (v.z == x1 && left > 2) k1 = k + 2;
            if (v.w == x0 && left > 3) k0 = k + 3;
            if (v.w == x1 && left > 3) k1 = k + 3;
        }
        if (k0 < 0) {
            k0 = append(x0, r0);
            if (x0 == x1) k1 = k0;
        }
        if (k1 < 0) k1 = append(x1, r1);
    }
    __device__ __forceinline__ int del(int k) {
        if (k < 0) return 0;
        const int s = sts[k * stride];
        sts[k * stride] = s | 8;
        return (s >> 1) & 1;
    }
    // the node's flag, or its fanins, matter to the candidate
    __device__ __forceinline__ void use_del(int k) {
        if (k >= 0) sts[k * stride] |= 8;
    }
    __device__ __forceinline__ void use_fanins(int k) {
        if (k >= 0) sts[k * stride] |= 32;
    }
    // whether the node's count, now v, is zero matters
    __device__ __forceinline__ void decide(int k, int v) {
        if (k < 0) return;
        const int s = sts[k * stride];
        if (v <= 0)
            sts[k * stride] = s | 16;
        else if (v < ((s >> 6) & kNoLow) || ((s >> 6) & kNoLow) == kNoLow)
            sts[k * stride] = (s & ~(kNoLow << 6)) | (min(v, kNoLow - 1) << 6);
    }
    __device__ __forceinline__ int ref(int k, int base) const { return k >= 0 ? base + (sts[k * stride] >> 16) : base; }
    __device__ __forceinline__ void add(int k, int d) {
        if (k >= 0) sts[k * stride] += d * 65536;
    }
    __device__ __forceinline__ void set_del(int k, int v) { sts[k * stride] = (sts[k * stride] & ~2) | (v << 1) | 8; }
    __device__ __forceinline__ void set_fanins(int k, int, int) { sts[k * stride] |= 4; }
    __device__ __forceinline__ bool failed() const { return full; }
    // whether the flag of the node of state st ends up changed
    static __device__ __forceinline__ bool flipped(int st) { return (st ^ (st >> 1)) & 1; }
    // Whether a candidate at place t that holds state st of a node saw it stale,
    // given the node's marks.  A count that mattered as positive still is when
    // it exceeds all that the window's other candidates take away.
    static __device__ __forceinline__ bool stale(int st, const int4 &mark, int t) {
        const int low = (st >> 6) & kNoLow, own = st >> 16;
        return ((st & 8) && mark.x < t) || ((st & 32) && mark.w < t) ||
               (mark.y < t && ((st & 16) || (low < kNoLow && low <= mark.z - (own < 0 ? -own : 0))));
    }
};

// Traversal stacks.  Frames: FastDelete's {handle, count << 2 | where to
// resume (1: at fanin 1, 2: at the end), fanin0 literal, fanin1 literal},
// install's {handle, 0, fanin0 literal, fanin1 literal}.
struct GraphStack {
    int4 *s;
    int cap;
    int *status;
    bool full;
    __device__ __forceinline__ void push(int &sp, int4 f) {
        if (sp + 1 >= cap) {
            set_status(status, kDevStackOverflow);
            full = true;
            return;
        }
        s[sp++] = f;
    }
    __device__ __forceinline__ int4 pop(int &sp) const { return s[--sp]; }
};

// (the frames are an array of their own, so that the walk's scalars beside
// them stay in registers)
struct SpecStack {
    int4 *s;
    bool full;
    __device__ __forceinline__ void push(int &sp, int4 f) {
        if (sp >= kSpecFrames) {
            full = true;
            return;
        }
        s[sp++] = f;
    }
    __device__ __forceinline__ int4 pop(int &sp) const { return s[--sp]; }
};

// One candidate of the choice loop (rewrite.cu:849-897), replayed one
// traversed node per step, so that the lanes of a warp, each with a candidate
// of its own, take every node's loads together (as nested loops the lanes
// drifted apart and a window's replays ran one lane at a time: 80 us a round
// instead of 9).
//
// install (rewrite.cu:835-847): whether a node is installed depends only on
// the deletion flags, which the walk clears as it reaches nodes, and install
// reads no reference count, so every visiting order installs the same nodes,
// makes the same increments and returns the same count: a worklist (a node's
// deleted fanins are cleared and queued when the node is taken) instead of
// the recursion.
//
// FastDelete (rewrite.h:208-220): the recursion with an explicit stack.  A
// node is opened (both fanins' decrements), then its fanin 0 entered if its
// count fell to zero, then -- with fanin 1's count read again, since fanin
// 0's subtree may have changed it -- its fanin 1, then it is marked deleted
// and its count handed to its parent.
template <class Mem, class Stack>
struct Replay {
    Mem m;
    Stack st;
    int trueLit;
    int64_t nL0;
    int useZeros;
    // the candidate: its node and replacement, their handles and fanins
    int rep, kq, q0, q1, kn, n0, n1, nRef;
    // the walk
    enum Mode { kInstall, kOpen, kRecheck };
    int phase, mode, k, l0, l1, cnt, sp;
    int added, gain, code;
    bool busy;

    __device__ __forceinline__ int red(int a, int b) const { return a == b || a == trueLit; }

    __device__ __forceinline__ void begin_install(int h, int a, int b) {
        m.set_del(h, 0);
        mode = kInstall, k = h, l0 = a, l1 = b, cnt = 0, sp = 0;
    }
    __device__ __forceinline__ void begin_delete(int h, int a, int b) { mode = kOpen, k = h, l0 = a, l1 = b, sp = 0; }
    __device__ __forceinline__ void done(int c) {
        code = c;
        busy = false;
    }

    // a = {c, q, rep, -}, lv the cut's leaves
    __device__ __forceinline__ void start(int4 a, int4 lv) {
        const int q = a.y;
        rep = a.z;
        const int x = rep >> 1;
        const int4 rn = m.ld(x), rq = m.ld(q);
        const int4 r0 = m.ld(lv.x), r1 = m.ld(lv.y), r2 = m.ld(lv.z), r3 = m.ld(lv.w);
        busy = true;
        gain = 0;
        n0 = rn.x, n1 = rn.y, nRef = rn.z, q0 = rq.x, q1 = rq.y;
        // the leaves are distinct nodes below q; the replacement may be one
        m.use_del(m.append(lv.x, r0));
        m.use_del(m.append(lv.y, r1));
        m.use_del(m.append(lv.z, r2));
        m.use_del(m.append(lv.w, r3));
        m.slots(q, rq, x, rn, kq, kn);
        m.use_fanins(kq);
        m.use_fanins(kn);
        if (x == q || (n1 >> 1) == q) return done(kChSelfRef);
        if (r0.w | r1.w | r2.w | r3.w) return done(kChCompromised);
        phase = 0;
        if (m.del(kn))
            begin_install(kn, n0, n1);
        else
            finish(0);
    }

    // the walk of the current phase ended with count c
    __device__ __forceinline__ void finish(int c) {
        if (phase == 0) {  // the replacement is installed: delete the node
            added = c;
            m.add(kn, 1);
            phase = 1;
            return begin_delete(kq, q0, q1);
        }
        if (phase == 1) {
            m.add(kn, -1);
            gain = c - added;
            if (gain > 0 || (gain == 0 && useZeros)) {
                m.set_del(kq, 0);
                m.set_fanins(kq, trueLit, rep);
                m.add(kn, 1);
                return done(kChCommitted);
            }
            phase = 2;
            if (m.del(kq)) return begin_install(kq, q0, q1);
        }
        if (phase == 2) {  // the node is back: drop the replacement
            m.add(kq, 1);
            phase = 3;
            const int v = m.ref(kn, nRef);
            m.decide(kn, v);
            if (kn >= 0 && v == 0) return begin_delete(kn, n0, n1);
        }
        m.add(kq, -1);
        done(kChReverted);
    }

    // one node of the walk
    __device__ __forceinline__ void step() {
        const int c0 = l0 >> 1, c1 = l1 >> 1;
        const int4 r0 = m.ld(c0), r1 = m.ld(c1);
        int k0, k1;
        m.slots(c0, r0, c1, r1, k0, k1);
        if (mode == kInstall) {
            cnt += 1 - red(l0, l1);
            const int d0 = m.del(k0), d1 = m.del(k1);
            m.add(k0, 1);
            m.add(k1, 1);
            if (d1 && c1 != c0) {
                m.set_del(k1, 0);
                m.use_fanins(k1);
                st.push(sp, make_int4(k1, 0, r1.x, r1.y));
            }
            if (d0) {
                m.set_del(k0, 0);
                m.use_fanins(k0);
                k = k0, l0 = r0.x, l1 = r0.y;
            } else if (sp > 0) {
                const int4 f = st.pop(sp);
                k = f.x, l0 = f.z, l1 = f.w;
            } else {
                finish(cnt);
            }
        } else {
            int v0 = 1, v1;
            if (mode == kOpen) {
                cnt = 1 - red(l0, l1);
                const int o0 = m.ref(k0, r0.z);
                m.add(k0, -1);
                v1 = m.ref(k1, r1.z) - 1;
                m.add(k1, -1);
                v0 = c0 == c1 ? v1 : o0 - 1;  // one node twice: both decrements precede the first check
                m.decide(k0, v0);
            } else {
                v1 = m.ref(k1, r1.z);
            }
            m.decide(k1, v1);
            if (v0 == 0 && k0 >= 0) {
                st.push(sp, make_int4(k, (cnt << 2) | 1, l0, l1));
                m.use_fanins(k0);
                mode = kOpen, k = k0, l0 = r0.x, l1 = r0.y;
            } else if (v1 == 0 && k1 >= 0) {
                st.push(sp, make_int4(k, (cnt << 2) | 2, l0, l1));
                m.use_fanins(k1);
                mode = kOpen, k = k1, l0 = r1.x, l1 = r1.y;
            } else {
                while (true) {
                    m.set_del(k, 1);
                    if (sp == 0) {
                        finish(cnt);
                        break;
                    }
                    const int4 f = st.pop(sp);
                    k = f.x, l0 = f.z, l1 = f.w;
                    cnt += f.y >> 2;
                    if ((f.y & 3) == 1) {
                        mode = kRecheck;
                        break;
                    }
                }
            }
        }
        if (m.failed() || st.full) busy = false;
    }
};

// Rounds of a window of candidates, one per thread (see the top of the
// file); T threads on each of B blocks (a cluster when B > 1), the window's
// places dealt to the warps in turn.  A round is three barriers: every thread
// replays its candidate and marks each node it changes with its place in the
// window; a thread that saw one of its nodes stale must wait, and the lowest
// such place ends the part that is committed; committing adds the overlay's
// changes to the records.  Flags and fanins that a committed candidate changes,
// no later committed one has used; counts change by sums.  A candidate that
// outgrows its overlay ends the window and, at its start, is replayed by thread
// 0 on the committed graph.  The next window is up to four times the part
// committed, at least two places a warp.
//
// Where candidates depend on one another in a row -- the stages of a ripple
// carry chain, whose every replacement changes what the next one reads -- a
// window commits hardly more than one of them.  After a window that committed
// fewer than kFew, thread 0 replays the next ones on the committed graph: two
// of them, and twice as many after each further such window.
//
// Bound: the latency of a replay's dependent record loads (about ten), 10-16
// us a round, 2 us for a candidate replayed alone, whose records are in L1.
// One thread walking the candidates took 2.3-2.5 us for each. 64x64 multiplier
// (4,157 candidates, 61 committed at a time; 25 when every change of a node
// made it stale): 9.6 -> 0.76 ms; 1M-AND layered graph with rw -z (80,251
// tried, 345 at a time): 202 -> 3.7 ms; 256 graphs of up to 200k ANDs: 15.1 ->
// 2.5 ms.  A ripple carry adder of 4,000 bits, rw -z: 29 ms by one thread, 135
// in windows alone, 24 now; 300 of 64 bits: 0.79, 4.03, 0.92.
template <int T, int B>
__global__ void __launch_bounds__(T, 1) k_choice(ChoiceArgs A) {
    using Overlay = OverlayMem<B == 1>;
    extern __shared__ int4 s_overlay[];
    __shared__ int s_stop[2];
    constexpr int kWarps = T / 32 * B;
    constexpr int kFew = B == 1 ? 4 : 8;  // a round's time over a replay's
    const int tid = threadIdx.x, g = blockIdx.x / B, rank = blockIdx.x % B;
    const int t = (tid & 31) * kWarps + rank * (T / 32) + (tid >> 5);  // place in the window
    auto barrier = [] {
        if (B == 1)
            __syncthreads();
        else
            cg::this_cluster().sync();
    };
    int *stops = B == 1 ? s_stop : cg::this_cluster().map_shared_rank(s_stop, 0);
    const int64_t nL0 = A.nL0;
    const int trueLit = 2 * A.dg[g].cpos + 1;
    int base = gridDim.x > B ? A.gStart[g] : 0;
    const int end = gridDim.x > B ? base + A.gCount[g] : A.n;
    if (tid < 2) s_stop[tid] = INT_MAX;
    barrier();
    int nDone[kChReverted + 1] = {}, nPos = 0, expected = 0;
    int window = A.serial ? 1 : T * B, alone = 0;
    for (int round = 0; base < end; round++) {
        const int nAct = min(window, end - base);
        const bool act = t < nAct;
        int *stop = &stops[round & 1];
        Replay<Overlay, SpecStack> R;
        int4 frames[kSpecFrames];
        R.m = Overlay{A.rec, nL0, s_overlay + tid, reinterpret_cast<int *>(s_overlay + kOverlay / 4 * T) + tid, T, 0, false};
        R.st = SpecStack{frames, false};
        R.trueLit = trueLit;
        R.nL0 = nL0;
        R.useZeros = A.useZeros;
        R.busy = false;
        int4 a = make_int4(-1, -1, -1, -1);
        if (act) {
            a = A.recA[base + t];
            R.start(a, A.recB[base + t]);
        }
        while (__any_sync(0xffffffffu, R.busy)) {
            if (R.busy) R.step();
            __syncwarp();
        }
        const bool outgrown = R.m.full || R.st.full || A.serial;
        // the overlay's entries four at a time, so that their accesses overlap
        const int n = act && !outgrown ? R.m.n : 0;
        for (int k = 0; k < n; k += 4) {
            const int4 x = R.m.ids[(k >> 2) * T];
            const int node[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (k + j >= n) continue;
                const int st = R.m.sts[(k + j) * T], d = st >> 16;
                int4 *mark = &A.mark[node[j]];
                if (Overlay::flipped(st)) atomicMin(&mark->x, t);
                if (d) atomicMin(&mark->y, t);
                if (d < 0) atomicAdd(&mark->z, -d);
                if (st & 4) atomicMin(&mark->w, t);
            }
        }
        if (rank == 0 && tid == 0) s_stop[(round + 1) & 1] = INT_MAX;
        barrier();
        if (act) {
            bool wait = outgrown;
            for (int k = 0; k < n; k += 8) {
                int4 m[8];
                const int4 x = R.m.ids[(k >> 2) * T], y = R.m.ids[((k >> 2) + 1) * T];
                const int node[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
                for (int j = 0; j < 8; j++)
                    m[j] = k + j < n ? __ldcg(&A.mark[node[j]]) : make_int4(INT_MAX, INT_MAX, 0, INT_MAX);
#pragma unroll
                for (int j = 0; j < 8; j++) wait |= k + j < n && Overlay::stale(R.m.sts[(k + j) * T], m[j], t);
            }
            if (wait) atomicMin(stop, t);
        }
        barrier();
        const int done = min(*stop, nAct);
        for (int k = 0; k < n; k += 4) {
            const int4 x = R.m.ids[(k >> 2) * T];
            const int node[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (k + j >= n) continue;
                const int st = R.m.sts[(k + j) * T];
                if (!Overlay::flipped(st) && !(st >> 16) && !(st & 4)) continue;
                A.mark[node[j]] = make_int4(INT_MAX, INT_MAX, 0, INT_MAX);
                if (t >= done) continue;
                int4 *rec = A.rec + node[j];
                if (st >> 16) atomicAdd(&rec->z, st >> 16);
                if (Overlay::flipped(st)) rec->w = (st >> 1) & 1;
                if (st & 4) {
                    rec->x = trueLit;
                    rec->y = a.z;
                }
            }
        }
        auto count = [&](int c, int code, int gain) {
            A.choice[c] = code;
#pragma unroll
            for (int k = 0; k <= kChReverted; k++) nDone[k] += code == k;
            if (code == kChCommitted) {
                nPos += gain > 0;
                expected += gain;
            }
        };
        if (t < done) count(a.x, R.code, R.gain);
        base += done;
        // the next candidates alone: more and more while windows commit few
        alone = done >= nAct || done >= kFew ? 0 : min(max(2, 2 * alone), kMaxAlone);
        const int single = min(A.serial ? 1 : alone, end - base);
        window = A.serial ? 1 : min(T * B, max(2 * kWarps, 4 * done));
        if (single > 0) {
            barrier();
            if (t == 0) {
                Replay<GraphMem, GraphStack> S;
                S.m = GraphMem{A.rec, nL0};
                S.st = GraphStack{A.stack + (int64_t)g * A.stackCap, A.stackCap, A.status, false};
                S.trueLit = trueLit;
                S.nL0 = nL0;
                S.useZeros = A.useZeros;
                int4 na = A.recA[base], nb = A.recB[base];
                for (int k = base; k < base + single; k++) {
                    const int4 x = na, lv = nb;
                    if (k + 1 < base + single) {  // the next one's, while this one is replayed
                        na = A.recA[k + 1], nb = A.recB[k + 1];
                    }
                    S.code = kChNotVisited;
                    S.start(x, lv);
                    while (S.busy) S.step();
                    count(x.x, S.code, S.gain);
                }
            }
            base += single;
        }
        barrier();
    }
    const int tot[7] = {nDone[kChCommitted],   nPos,     nDone[kChCommitted] - nPos, nDone[kChReverted],
                        nDone[kChCompromised], nDone[kChSelfRef], expected};
#pragma unroll
    for (int k = 0; k < 7; k++) {
        const int v = __reduce_add_sync(0xffffffffu, tot[k]);
        if ((tid & 31) == 0 && v) atomicAdd(&A.stats[k], (unsigned long long)(long long)v);
    }
}

// Gathers the nodes' records and clears their marks.
__global__ void k_choice_pack(int64_t M, const int *L0, const int *L1, const int *ref, const uint8_t *del, int4 *rec,
                              int4 *mark) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < M; x += stride) {
        rec[x] = make_int4(L0[x], L1[x], ref[x], del[x]);
        mark[x] = make_int4(INT_MAX, INT_MAX, 0, INT_MAX);
    }
}

// The walk's result (the reference counts are not needed any more).
__global__ void k_choice_unpack(int64_t M, const int4 *rec, int *L0, int *L1, uint8_t *del) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < M; x += stride) {
        const int4 r = rec[x];
        L0[x] = r.x;
        L1[x] = r.y;
        del[x] = (uint8_t)r.w;
    }
}

// the choice's record of the i-th candidate in graph order: {c, q, rep, -}
// and the chosen cut's four leaves (the constant in the fourth place of a
// three-leaf cut)
__global__ void k_cand_records(int64_t n, const int *candByG, const int *cand, const int *repW, const int8_t *bestCut,
                               const int4 *cutL, const int2 *cutM, const int *wg, const DevGraph *dg, int4 *recA,
                               int4 *recB) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int c = candByG[i];
        const int q = cand[c];
        const int slot = bestCut[q];
        int4 l = cutL[(int64_t)q * 8 + slot];
        if (packed_nleaves((uint32_t)cutM[(int64_t)q * 8 + slot].y) == 3) l.w = dg[wg[q]].cpos;
        recA[i] = make_int4(c, q, repW[c], 0);
        recB[i] = l;
    }
}

// graph of the i-th candidate that has a replacement
__global__ void k_cand_gid(int64_t n, const int *withRep, const int *cand, const int *wg, uint32_t *keys, int *vals,
                           int *gCount) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int c = withRep[i];
        const int g = wg[cand[c]];
        keys[i] = (uint32_t)g;
        vals[i] = c;
        agg_add(gCount, g, 1);
    }
}

template <int T, int B>
cudaError_t launch_choice(const ChoiceArgs &A, int G, cudaStream_t s) {
    const int smem = 2 * kOverlay * T * (int)sizeof(int);  // ids and states
    cudaError_t e = cudaFuncSetAttribute(k_choice<T, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(G * B));
    cfg.blockDim = dim3(T);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = B;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = B > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_choice<T, B>, A);
}

}  // namespace

int rw_choice(ExecCtx &X, Batch &b, RwWork &w) {
    const int G = w.G;
    const int64_t nCand = w.nCand, nRep = w.nRep;
    const int64_t M = w.N + w.nNew;  // extent of L0, L1, ref, del
    cudaStream_t s = X.s;
    Arena &ar = *X.ar;
    int rc;
    int *gCount = ar.get<int>(G + 1), *gStart = ar.get<int>(G + 1), *candByG = ar.get<int>(nRep + 1);
    uint32_t *keys = ar.get<uint32_t>(nRep + 1), *keys2 = ar.get<uint32_t>(nRep + 1);
    int *vals = ar.get<int>(nRep + 1);
    int4 *recA = ar.get<int4>(nRep + 1), *recB = ar.get<int4>(nRep + 1);
    w.choice = ar.get<int>(nCand + 1);
    unsigned long long *dstats = reinterpret_cast<unsigned long long *>(X.counters + kCtStats);
    // explicit recursion stacks: deep enough for any chain through the
    // levels plus the new nodes
    int64_t stackCap = (int64_t)w.maxLevel + 64;
    stackCap = std::min<int64_t>(2 * stackCap + w.nNew / std::max(G, 1) + 64, 1 << 20);
    int4 *stack = ar.get<int4>((size_t)stackCap * G);
    // the records and marks take the place of the enumeration's cuts, 256
    // bytes per original node, which are not read any more once the
    // candidates' records are made
    int4 *rec, *mark;
    if (32 * M <= 256 * w.N) {
        rec = w.cutL;
        mark = rec + M;
    } else {
        rec = ar.get<int4>(M);
        mark = ar.get<int4>(M);
    }
    if (!gCount || !gStart || !candByG || !keys || !keys2 || !vals || !recA || !recB || !w.choice || !stack ||
        !rec || !mark)
        return X.fail(CULS_E_OOM, "rw: arena exhausted (choice)");
    if (G > 1 && (rc = X.check(cudaMemsetAsync(gCount, 0, sizeof(int) * (G + 1), s), "memset"))) return rc;
    if ((rc = X.check(cudaMemsetAsync(dstats, 0, sizeof(unsigned long long) * 8, s), "memset"))) return rc;
    if ((rc = X.check(fill_i32(w.choice, kChNoReplace, nCand, s), "fill"))) return rc;
    if (nRep > 0) {
        if (G > 1) {
            k_cand_gid<<<X.grid(nRep), kBlock, 0, s>>>(nRep, w.withRep, w.cand, w.wg, keys, vals, gCount);
            X.launched(1);
            int bits = 1;
            while ((1ll << bits) < G) bits++;
            if ((rc = X.check(radix_sort_pairs(keys, vals, keys2, candByG, nRep, bits, ar, s), "sort"))) return rc;
            if ((rc = X.check(scan_exclusive(gCount, gStart, G, nullptr, ar, s), "scan"))) return rc;
        } else {
            candByG = w.withRep;
        }
        k_cand_records<<<X.grid(nRep), kBlock, 0, s>>>(nRep, candByG, w.cand, w.repW, w.bestCut, w.cutL, w.cutM, w.wg,
                                                       w.dg, recA, recB);
        k_choice_pack<<<X.grid(M), kBlock, 0, s>>>(M, w.L0, w.L1, w.ref, w.del, rec, mark);
        // CULS_CHOICE_GLOBAL replays every candidate alone (the tests compare
        // the two)
        ChoiceArgs A{w.nL0,  w.dg,  rec,           mark,     recA,   recB,    gStart, gCount, (int)nRep, w.useZeros ? 1 : 0,
                     getenv("CULS_CHOICE_GLOBAL") ? 1 : 0, stack, (int)stackCap, w.choice, dstats, X.status};
        // Threads per graph: a cluster of eight SMs for few graphs of many
        // candidates (not on an SM partition, whose SMs need not hold a whole
        // cluster), so that the replays of a window share no SM's load path
        // (1M-AND rw -z 4.6 -> 3.7 ms, 64x64 multiplier 0.87 -> 0.76; its
        // barriers cost more where 95 candidates are all there are: 0.28 ->
        // 0.31); else a window as wide as an SM's shared memory allows while
        // there is an SM for every graph, narrower ones so that more graphs
        // are resident when there are more (a batch's graphs have short
        // windows: 7 candidates are committed at a time in 256 graphs of up to
        // 200k ANDs, 345 in the 1M-AND graph).
        if (X.clusters && 8 * G <= X.sms && nRep >= 1024 * (int64_t)G)
            rc = X.check(launch_choice<128, 8>(A, G, s), "choice launch");
        else if (G <= X.sms)
            rc = X.check(launch_choice<512, 1>(A, G, s), "choice launch");
        else if (G <= 3 * X.sms)
            rc = X.check(launch_choice<256, 1>(A, G, s), "choice launch");
        else
            rc = X.check(launch_choice<64, 1>(A, G, s), "choice launch");
        if (rc) return rc;
        k_choice_unpack<<<X.grid(M), kBlock, 0, s>>>(M, rec, w.L0, w.L1, w.del);
        X.launched(4);
    }
    (void)b;
    return 0;
}

namespace {

// per node, fixed during the sweeps
enum : uint8_t { kRdPi = 1, kRdDel = 2, kRdR0 = 4 };  // PI or constant; deleted; redundant before the sweep

struct RedArgs {
    int64_t M;
    const int *gidAll;
    const DevGraph *dg;
    const int *pre0, *pre1;
    const uint8_t *st;
    const int *postIn1;
    const uint8_t *nredIn;
    int *post1;
    uint8_t *nredOut;
    int *changed;
    int *status;
};

__global__ void k_red_state(int64_t M, int64_t nL0, const int *gidAll, const DevGraph *dg, const int *L0, const int *L1,
                            const uint8_t *del, uint8_t *st) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < M; x += stride) {
        if (x < nL0) {
            st[x] = kRdPi;
            continue;
        }
        const int a = L0[x];
        const bool r0 = a == L1[x] || a == 2 * dg[gidAll[x]].cpos + 1;
        st[x] = (uint8_t)((del[x] ? kRdDel : 0) | (r0 ? kRdR0 : 0));
    }
}

// Fanin() of rewrite.h:121-124 as seen by the sweep at node `time`
// (time = INT_MAX after the sweep).  A node is chased (its fanins are
// rewritten by the sweep) when it is no PI, not deleted and not redundant
// before the sweep: state byte 0.
__device__ int rd_chase(const RedArgs &A, int lit, int time) {
    int c = 0;
    for (int step = 0; step < (1 << 20); step++) {
        const int u = lit >> 1;
        const int s = A.st[u];
        if (s & kRdPi) return lit ^ c;
        const bool done = u < time && s == 0;
        const bool red = done ? A.nredIn[u] != 0 : (s & kRdR0) != 0;
        if (!red) return lit ^ c;
        c ^= lit & 1;
        lit = done ? A.postIn1[u] : A.pre1[u];
    }
    set_status(A.status, kDevBadGraph);
    return lit ^ c;
}

// one sweep over the chased nodes; the others keep their fanins and are
// never read as sweep state
__global__ void k_redundancy(RedArgs A) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < A.M; x += stride) {
        if (A.st[x]) continue;
        const int a = rd_chase(A, A.pre0[x], (int)x);
        const int b = rd_chase(A, A.pre1[x], (int)x);
        const int t = 2 * A.dg[A.gidAll[x]].cpos + 1;
        const uint8_t nr = (a == b || a == t) ? 1 : 0;
        if (nr != A.nredIn[x] || b != A.postIn1[x]) atomicExch(A.changed, 1);
        A.post1[x] = b;
        A.nredOut[x] = nr;
    }
}

// pre0 aliases L0 (each node reads and writes only its own entry); pre1 is a
// copy, since other nodes' chases read it
__global__ void k_redundancy_finish(RedArgs A, int *L0, int *L1, uint8_t *delOut, int64_t nPO, int *po) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < A.M; x += stride) {
        const int s = A.st[x];
        if (s == 0) {
            L0[x] = rd_chase(A, A.pre0[x], (int)x);
            L1[x] = A.postIn1[x];
        } else if (!(s & (kRdPi | kRdDel))) {
            delOut[x] = 1;  // redundant before the sweep: rewrite.cu:916-917
        }
    }
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < nPO; k += stride) po[k] = rd_chase(A, po[k], INT_MAX);
}

}  // namespace

int rw_redundancy(ExecCtx &X, Batch &b, RwWork &w, RwStats *stats) {
    (void)b;
    const int64_t M = w.N + w.nNew;
    cudaStream_t s = X.s;
    Arena &ar = *X.ar;
    int rc;
    int *pre1 = ar.get<int>(M);
    int *P1[2] = {ar.get<int>(M), ar.get<int>(M)};
    uint8_t *NR[2] = {ar.get<uint8_t>(M), ar.get<uint8_t>(M)};
    uint8_t *st = ar.get<uint8_t>(M);
    if (!pre1 || !P1[0] || !P1[1] || !NR[0] || !NR[1] || !st) return X.fail(CULS_E_OOM, "rw: arena exhausted (redundancy)");
    if ((rc = X.check(cudaMemcpyAsync(pre1, w.L1, sizeof(int) * M, cudaMemcpyDeviceToDevice, s), "copy"))) return rc;
    if ((rc = X.check(cudaMemsetAsync(NR[0], 0, M, s), "memset"))) return rc;
    k_red_state<<<X.grid(M), kBlock, 0, s>>>(M, w.nL0, w.gidAll, w.dg, w.L0, w.L1, w.del, st);
    X.launched(1);
    int *changed = X.counters + 24;
    // sweep state: (post1, nred) of the chased nodes; state 0 (no chase
    // yet) is (pre1, 0), read from pre1 itself.  Two sweeps per host check:
    // the second one usually finds nothing left to change.
    const int *in1 = pre1;
    const uint8_t *inR = NR[0];
    int cur = 1;
    for (int it = 0;; it += 2) {
        if (it >= 64) return X.fail(CULS_E_INVALID, "rw: redundancy sweep did not converge");
        if ((rc = X.check(cudaMemsetAsync(changed, 0, sizeof(int) * 2, s), "memset"))) return rc;
        for (int k = 0; k < 2; k++) {
            RedArgs A{M, w.gidAll, w.dg, w.L0, pre1, st, in1, inR, P1[cur], NR[cur], changed + k, X.status};
            k_redundancy<<<X.grid(M), kBlock, 0, s>>>(A);
            in1 = P1[cur];
            inR = NR[cur];
            cur ^= 1;
        }
        X.launched(2);
        if ((rc = X.fetch("rw choice and redundancy"))) return rc;
        if (!X.hostSmall[25]) break;
    }
    // (in1, inR) is a fix-point: sweeping it again reproduces it
    RedArgs F{M, w.gidAll, w.dg, w.L0, pre1, st, in1, inR, nullptr, nullptr, changed, X.status};
    k_redundancy_finish<<<X.grid(std::max<int64_t>(M, w.nPO)), kBlock, 0, s>>>(F, w.L0, w.L1, w.del, w.nPO, w.wpo);
    X.launched(1);
    if (stats) {
        const int64_t nAnd = w.N - w.nL0, nCand = w.nCand, nRep = w.nRep;
        unsigned long long hs[8], warpPairs;
        memcpy(hs, X.hostSmall + kCtStats, sizeof hs);
        memcpy(&warpPairs, X.hostSmall + kCtPairs, sizeof warpPairs);
        stats->replaced = (long long)hs[0];
        stats->replacedPos = (long long)hs[1];
        stats->replacedZero = (long long)hs[2];
        stats->reverted = (long long)hs[3];
        stats->compromised = (long long)hs[4];
        stats->newIdx = nCand - nRep;
        stats->expected = (long long)hs[6];
        stats->preEval = nAnd - nCand;
        stats->smallCut = 0;
        stats->newNodes = w.nNew;
        stats->candidates = nCand;
        stats->warpPairs = (long long)warpPairs;
    }
    return 0;
}

}  // namespace culs
