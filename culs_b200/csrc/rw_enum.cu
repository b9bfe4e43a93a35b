// 4-input cut enumeration with 16-bit truth tables: the B200 form of
// Inputs + CutEnumerate (CULS src/algorithms/rewrite.cu:63-74,268-294).
//
// The reference launches one kernel per level (rewrite.cu:703-704).  Here a
// run of levels of like width is one launch of a persistent dataflow kernel,
// which walks the level-major layout in order: a node waits (bounded) until
// both fanins have published their cut sets, and the reference's per-pair slot
// policy is replayed exactly.  Wide levels take a node per thread
// (k_enumerate), with the 8 slots in registers (fully unrolled slot loops);
// narrower ones a node per warp (k_enumerate_warp), which builds the candidate
// cuts of all pairs side by side.  Every cut record carries its leaves'
// reference counts and local-id bits (cutA), so a node reads nothing but its
// two fanins' 16 cut records.  Pairs whose 32-bit signatures already exceed 4
// leaves are rejected from the fanins' {sign, packed} words before any leaf
// data is used.
#include <algorithm>
#include <vector>

#include "enum_regs.cuh"
#include "rw_work.cuh"

namespace culs {

namespace {

constexpr int kEnumBlock = 128;

struct EnumArgs {
    int64_t q0, q1;         // the W positions of the launch's levels
    int nLevels;            // its levels,
    const int *lvlStart;    //   the first W position of each and the end (nLevels + 1 entries), and
    const int *chunkStart;  //   the first 32-node chunk of each and the end
    const int *w0, *w1;
    const int *ref;
    const uint8_t *lidLow;
    int4 *cutL;
    int2 *cutM;
    int2 *cutA;
    int *done;
    int *counter;
    unsigned long long *warpPairs;  // pairs replayed by enum_node_warp
    int *status;
};

__device__ __forceinline__ uint32_t leaf_attr(int ref, uint32_t lid) {
    return (ref > 1001 ? 1001u : (uint32_t)ref) | ((lid & 31u) << 11);
}

__global__ void k_enum_init(int64_t N, const int *wlev, const int *wl, const uint8_t *lidLow, const int *ref,
                            int4 *cutL, int2 *cutM, int2 *cutA, int *done) {
    int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < N; q += stride) {
        bool lev0 = wlev[q] == 0;
        done[q] = lev0 ? 1 : 0;
        if (lev0 && wl[q] != 0) {  // primary input: the trivial cut only
            Cut c;
            c.sign = 1u << lidLow[q];
            c.tt = 0xAAAAu;
            c.nLeaves = 1;
            c.used = 1;
            c.value = 1001u;  // CutFindValue of a one-leaf cut
            cutL[q * 8] = make_int4((int)q, 0, 0, 0);
            cutM[q * 8] = make_int2((int)c.sign, (int)cut_pack(c));
            cutA[q * 8] = make_int2((int)leaf_attr(ref[q], lidLow[q]), 0);
        }
    }
}

// A slot in registers: leaves, signature, packed tt/value/nLeaves/used.  The
// slot's aux word is written straight to cutA when the slot is filled: this
// node never reads it back.
struct Slot {
    int l[4];
    uint32_t sign, pk;
};

__device__ __forceinline__ uint32_t sl_n(const Slot &s) { return packed_nleaves(s.pk); }
__device__ __forceinline__ uint32_t sl_used(const Slot &s) { return packed_used(s.pk); }
__device__ __forceinline__ uint32_t sl_value(const Slot &s) { return (s.pk >> 16) & 0x7FFu; }
__device__ __forceinline__ void sl_clear_used(Slot &s) { s.pk &= ~(1u << 30); }

// every leaf of (al, an) appears among the leaves of (bl, bn)
__device__ __forceinline__ bool leaves_subset(const int (&al)[4], uint32_t an, const int (&bl)[4], uint32_t bn) {
    bool all = true;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        bool in = false;
#pragma unroll
        for (int j = 0; j < 4; j++) in |= ((uint32_t)j < bn) && bl[j] == al[i];
        all &= ((uint32_t)i >= an) || in;
    }
    return all;
}

// CutFilter (rewrite.cu:178-193) for the cut X sitting in slot id: visits the
// other used slots in index order, drops larger slots that contain X and
// stops (dropping X) at the first slot contained in X.
__device__ __forceinline__ bool filter_slots(Slot (&S)[8], int id, const int (&xl)[4], uint32_t xn, uint32_t xs) {
    bool dropped = false;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        if (dropped || k == id || !sl_used(S[k])) continue;
        const uint32_t kn = sl_n(S[k]);
        if (kn > xn) {
            if ((S[k].sign & xs) == xs && leaves_subset(xl, xn, S[k].l, kn)) sl_clear_used(S[k]);
        } else {
            if ((S[k].sign & xs) == S[k].sign && leaves_subset(S[k].l, kn, xl, xn)) dropped = true;
        }
    }
    return dropped;
}

__device__ __forceinline__ void load_rcut(const EnumArgs &A, int64_t idx, int2 m, RCut &c) {
    int4 l = A.cutL[idx];
    int2 x = A.cutA[idx];
    c.l[0] = l.x;
    c.l[1] = l.y;
    c.l[2] = l.z;
    c.l[3] = l.w;
    c.sign = (uint32_t)m.x;
    c.tt = (uint32_t)m.y & 0xFFFFu;
    c.n = packed_nleaves((uint32_t)m.y);
    c.used = 1;
    rc_unpack_aux((uint32_t)x.x, (uint32_t)x.y, c);
}

// ------------------------------------------------- warp-per-node variant
// A warp's scratch: its node's fanin cuts and candidates, one per admissible
// pair.
struct WarpCands {
    int4 leaves[64];  // final leaves
    int4 rec[64];     // final {sign, packed tt / value / nLeaves / used, cutA words}
    uint4 rel[64];    // the merged cut against earlier candidates' final cuts
    uint4 relMin[64]; // the same for the final cut, where minimisation removed leaves
    int4 inL[16], inR[16];  // the fanins' cuts: leaves, {sign, packed, cutA words}
    uint8_t pair[64]; // the k-th admissible pair
};

// How cut X stands to the final cuts of candidates 0 .. n - 1 (n <= 64), one
// bit each: {contained in X: 0-31, larger than X and containing it: 0-31,
// contained: 32-63, containing: 32-63}.  A cut's leaves are distinct, so the
// number of equal pairs of leaves decides containment either way; unused
// places are -1 in X and 0 in the candidates, which no leaf equals (position
// 0 is a constant, which has no cuts).  CutFilter's signature tests
// (rewrite.cu:178-193) follow from containment, as a cut's signature is the
// union of its leaves' bits.
// With at most 16 candidates, lane and lane + 16 hold the same X and take half
// of them each.
__device__ __forceinline__ uint4 relate(const WarpCands &W, int n, int lane, const int (&l)[4], uint32_t xn) {
    uint4 r = make_uint4(0, 0, 0, 0);
    const int x0 = xn > 0 ? l[0] : -1, x1 = xn > 1 ? l[1] : -1, x2 = xn > 2 ? l[2] : -1, x3 = xn > 3 ? l[3] : -1;
    const bool split = n <= 16;
    for (int h = 0; h < n; h += 32) {
        uint32_t sub = 0, sup = 0;
        const int e = n - h < 32 ? n - h : 32, half = (e + 1) >> 1;
        const int mEnd = split && lane < 16 ? half : e;
#pragma unroll 2
        for (int m = split && lane >= 16 ? half : 0; m < mEnd; m++) {
            const int4 y = W.leaves[h + m];
            const uint32_t yn = packed_nleaves((uint32_t)W.rec[h + m].y);
            uint32_t c = 0;
            c += (y.x == x0) + (y.x == x1) + (y.x == x2) + (y.x == x3);
            c += (y.y == x0) + (y.y == x1) + (y.y == x2) + (y.y == x3);
            c += (y.z == x0) + (y.z == x1) + (y.z == x2) + (y.z == x3);
            c += (y.w == x0) + (y.w == x1) + (y.w == x2) + (y.w == x3);
            sub |= (c == yn ? 1u : 0u) << m;
            sup |= (c == xn && yn > xn ? 1u : 0u) << m;
        }
        if (split) {
            sub |= __shfl_xor_sync(0xffffffffu, sub, 16);
            sup |= __shfl_xor_sync(0xffffffffu, sup, 16);
        }
        if (h == 0)
            r.x = sub, r.y = sup;
        else
            r.z = sub, r.w = sup;
    }
    // bit 63 stands for the node's trivial cut (candidate 63 has no successor
    // to compare it with): only an empty cut is related to it
    r.z &= 0x7FFFFFFFu;
    r.w = (r.w & 0x7FFFFFFFu) | (xn == 0 ? 1u << 31 : 0u);
    return r;
}

// CutFilter (rewrite.cu:178-193) over the slots in `used`, the cuts related
// to X by r, slot `lane` holding candidate c: visiting the slots in index
// order, a larger slot containing X is dropped and the first slot contained
// in X drops X and ends the visit -- so only the supersets before it are
// dropped.  Returns true when X is dropped.
__device__ __forceinline__ bool filter_related(uint4 r, int c, uint32_t among, uint32_t &used) {
    const uint32_t sub = (c & 32) ? r.z : r.x, sup = (c & 32) ? r.w : r.y;
    const uint32_t D = __ballot_sync(0xffffffffu, (sub >> (c & 31)) & 1u) & among;
    const uint32_t C = __ballot_sync(0xffffffffu, (sup >> (c & 31)) & 1u) & among;
    used &= ~(D ? C & ((D & (0u - D)) - 1u) : C);
    return D != 0;
}

// FindCut's order among full slots: class by leaves, then value.
__device__ __forceinline__ uint32_t slot_key(uint32_t pk) {
    const uint32_t n = packed_nleaves(pk);
    return ((n > 2 ? 0u : (n == 2 ? 1u : 2u)) << 20) | (((pk >> 16) & 0x7FFu) << 3);
}

// The fanin cut in place i.
__device__ __forceinline__ void fetch_slot(const WarpCands &W, int i, RCut &c) {
    const int4 L = W.inL[i], R = W.inR[i];
    c.l[0] = L.x;
    c.l[1] = L.y;
    c.l[2] = L.z;
    c.l[3] = L.w;
    c.sign = (uint32_t)R.x;
    c.tt = (uint32_t)R.y & 0xFFFFu;
    c.n = packed_nleaves((uint32_t)R.y);
    c.used = 1;
    rc_unpack_aux((uint32_t)R.z, (uint32_t)R.w, c);
}

// A warp enumerates one node at a time: lanes 0-7 hold u0's cut slots and
// lanes 8-15 u1's.  The admissible pairs (pair bit i * 8 + j, the reference's
// i-major order; both slots used, at most four leaves by signature) are
// listed in order and dealt out, the k-th to lane k % 32, so a node with at
// most 32 of them -- most nodes -- builds its candidates in one round.  The
// lanes then compare their candidates with all earlier ones, which turns
// CutEnumerate's slot policy, the sequential part, into a few bit operations
// a pair: slot s on lane s names the candidate it holds, the used slots are
// a mask in every lane, FindCut is its first clear bit or a min over the
// slots, CutFilter two ballots of precomputed bits.
//
// Bound: the node's latency on a narrow level, of which building the
// candidates takes 1.9 us, comparing them 1.0, the policy 1.6 (0.11 a pair)
// and publishing 1.2.  With the leaves compared inside the policy loop a pair
// took 0.18 us (0.38 while acquire polls slowed it) and the 64x64 multiplier
// (15 pairs a node, 501 levels) 15.9 us a level; now 8.4.
__device__ __forceinline__ void enum_node_warp(const EnumArgs &A, int64_t q, int lane, WarpCands &W) {
    const unsigned F = 0xffffffffu;
    constexpr int kTrivial = 64 + 63;  // the trivial cut's index: bit 63 of the relations
    const int f0 = A.w0[q], f1 = A.w1[q];
    const int u0 = f0 >> 1, u1 = f1 >> 1, c0 = f0 & 1, c1 = f1 & 1;
    int4 sl = make_int4(0, 0, 0, 0), sr = make_int4(0, 0, 0, 0);
    if (lane == 0) {  // slot 0: the trivial cut
        Cut c;
        c.sign = 1u << A.lidLow[q];
        c.tt = 0xAAAAu;
        c.nLeaves = 1;
        c.used = 1;
        c.value = 1001u;
        sl.x = (int)q;
        sr = make_int4((int)c.sign, (int)cut_pack(c), (int)leaf_attr(A.ref[q], A.lidLow[q]), 0);
    }
    int ok = 1;
    if (lane < 2) ok = wait_ge(&A.done[lane ? u1 : u0], 1, A.status);
    ok = __all_sync(F, ok);
    __syncwarp();  // orders the other lanes' reads below behind lanes 0 and 1's waits, which a vote does not
    int held = lane == 0 ? kTrivial : -1;  // candidate in this lane's slot
    uint32_t used = 1;
    if (ok) {
        int4 L = make_int4(0, 0, 0, 0);
        int2 M = make_int2(0, 0), X = make_int2(0, 0);
        if (lane < 16) {
            const int64_t idx = (int64_t)(lane < 8 ? u0 : u1) * 8 + (lane & 7);
            M = __ldcg(&A.cutM[idx]);
            L = __ldcg(&A.cutL[idx]);
            X = __ldcg(&A.cutA[idx]);
            W.inL[lane] = L;
            W.inR[lane] = make_int4(M.x, M.y, X.x, X.y);
        }
        // admissible pairs from the signatures: pair lane (i = lane / 8)
        // and pair lane + 32 (i = 4 + lane / 8), both with j = lane % 8
        const uint32_t sign = packed_used((uint32_t)M.y) ? (uint32_t)M.x : 0xFFFFFFFFu;  // unused: never admissible
        const uint32_t sA = __shfl_sync(F, sign, lane >> 3), sB = __shfl_sync(F, sign, 4 + (lane >> 3)),
                       sJ = __shfl_sync(F, sign, 8 + (lane & 7));
        const bool adm0 = popc32(sA | sJ) <= 4, adm1 = popc32(sB | sJ) <= 4;
        const uint32_t b0 = __ballot_sync(F, adm0), b1 = __ballot_sync(F, adm1);
        const uint32_t below = (1u << lane) - 1u;
        const int n0 = __popc(b0), nPairs = n0 + __popc(b1);
        if (adm0) W.pair[__popc(b0 & below)] = (uint8_t)lane;
        if (adm1) W.pair[n0 + __popc(b1 & below)] = (uint8_t)(lane + 32);
        __syncwarp();
        // candidate k built by lane k % 32; merged cuts of both rounds kept
        // until every final cut is in shared memory
        int ml[2][4];
        uint32_t mn[2] = {0, 0}, flags[2] = {0, 0};  // flags: 1 merged, 2 minimised, 4 fewer than two leaves
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if (r * 32 >= nPairs) break;
            const int k = r * 32 + (nPairs <= 16 ? lane & 15 : lane);
            const int p = W.pair[k < nPairs ? k : 0];
            RCut a, b, m;
            fetch_slot(W, p >> 3, a);
            fetch_slot(W, 8 + (p & 7), b);
            int pa, pb;
            const bool merged = rc_merge(a, b, m, pa, pb);
#pragma unroll
            for (int i = 0; i < 4; i++) ml[r][i] = m.l[i];
            mn[r] = m.n;
            m.tt = rc_truth(a, b, c0, c1, pa, pb);
            const bool mini = rc_minimize(m);
            if (k < nPairs && (nPairs > 16 || lane < 16)) {
                flags[r] = (merged ? 1u : 0u) | (mini ? 2u : 0u) | (m.n < 2 ? 4u : 0u);
                Cut pc;
                pc.tt = m.tt;
                pc.nLeaves = m.n;
                pc.used = 1;
                pc.value = rc_value(m);
                uint32_t x0, x1;
                rc_pack_aux(m, x0, x1);
                W.leaves[k] = make_int4(m.l[0], m.l[1], m.l[2], m.l[3]);
                W.rec[k] = make_int4((int)m.sign, (int)cut_pack(pc), (int)x0, (int)x1);
            }
        }
        __syncwarp();
        uint64_t merged = 0, mini = 0, stop = 0;
#pragma unroll
        for (int r = 0; r < 2; r++) {
            if (r * 32 >= nPairs) break;
            const int k = r * 32 + (nPairs <= 16 ? lane & 15 : lane), n = r == 0 && nPairs > 32 ? 32 : nPairs;
            const uint4 rel = relate(W, n, lane, ml[r], mn[r]);
            if (k < nPairs) W.rel[k] = rel;
            merged |= (uint64_t)__ballot_sync(F, flags[r] & 1u) << (r * 32);
            const uint32_t mm = __ballot_sync(F, (flags[r] & 3u) == 3u);
            stop |= (uint64_t)__ballot_sync(F, flags[r] & 4u) << (r * 32);
            if (mm) {
                const int4 y = W.leaves[k < nPairs ? k : 0];
                const int yl[4] = {y.x, y.y, y.z, y.w};
                const uint4 rm = relate(W, n, lane, yl, packed_nleaves((uint32_t)W.rec[k < nPairs ? k : 0].y));
                if (k < nPairs) W.relMin[k] = rm;
                mini |= (uint64_t)mm << (r * 32);
            }
        }
        __syncwarp();
        // the slot policy, pair by pair
        uint32_t key = lane < 8 ? slot_key((uint32_t)sr.y) | (uint32_t)lane : 0xFFFFFFFFu;
        int k = 0;
        for (; k < nPairs; k++) {
            const uint4 rel = W.rel[k];
            const uint32_t pk = (uint32_t)W.rec[k].y;
            // FindCut (rewrite.cu:84-109): the first free slot, else the
            // lowest (class, value, index)
            const uint32_t freeSlots = ~used & 0xFFu;
            const int id = freeSlots ? __ffs(freeSlots) - 1 : (int)(__reduce_min_sync(F, key) & 7u);
            used &= ~(1u << id);
            if (!((merged >> k) & 1u)) continue;
            if (filter_related(rel, held, used, used)) continue;  // the slot stays free
            if (lane == id) {
                held = k;
                key = slot_key(pk) | (uint32_t)lane;
            }
            bool drop = false;
            if ((mini >> k) & 1u) drop = filter_related(W.relMin[k], held, used, used);
            if (!drop) used |= 1u << id;
            if ((stop >> k) & 1u) {  // enumeration of this node stops (rewrite.cu:291)
                k++;
                break;
            }
        }
        if (lane == 0 && k > 0) atomicAdd(A.warpPairs, (unsigned long long)k);  // pairs replayed
        if (held >= 0 && held != kTrivial) sl = W.leaves[held], sr = W.rec[held];
    }
    if (lane < 8) {
        if (!((used >> lane) & 1u)) sr.y &= ~(1 << 30);
        A.cutL[q * 8 + lane] = sl;
        A.cutM[q * 8 + lane] = make_int2(sr.x, sr.y);
        A.cutA[q * 8 + lane] = make_int2(sr.z, sr.w);
    }
    // orders the lanes' stores before lane 0's release, which publishes them;
    // also: every lane is done reading W before the next node overwrites it
    __syncwarp();
    if (lane == 0) st_release(&A.done[q], 1);
}

// One node on one thread (wide levels): the slots in registers, the
// admissible pairs visited in order.  All lanes of the warp call it (valid:
// the lane has a node) and run as many rounds as the lane with the most
// admissible pairs, one pair per round and back in step after each, so
// lanes that finish a pair early do not drift into later pairs alone.
__device__ __forceinline__ void enum_node_thread(const EnumArgs &A, int64_t q, bool valid) {
    Slot S[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        S[k].pk = 0;
        S[k].sign = 0;
        S[k].l[0] = S[k].l[1] = S[k].l[2] = S[k].l[3] = 0;
    }
    if (valid) {
        Cut c;
        c.sign = 1u << A.lidLow[q];
        c.tt = 0xAAAAu;
        c.nLeaves = 1;
        c.used = 1;
        c.value = 1001u;
        S[0].l[0] = (int)q;
        S[0].sign = c.sign;
        S[0].pk = cut_pack(c);
        A.cutA[q * 8] = make_int2((int)leaf_attr(A.ref[q], A.lidLow[q]), 0);
    }
    const int f0 = valid ? A.w0[q] : 0, f1 = valid ? A.w1[q] : 0;
    const int u0 = f0 >> 1, u1 = f1 >> 1, c0 = f0 & 1, c1 = f1 & 1;
    bool ok = valid && wait_ge(&A.done[u0], 1, A.status) && wait_ge(&A.done[u1], 1, A.status);
    uint64_t pairs = 0;
    const int2 *M0 = A.cutM + (int64_t)u0 * 8, *M1 = A.cutM + (int64_t)u1 * 8;
    if (ok) {
        // the pairs CutEnumerate tries (both slots used, at most 4 leaves
        // by signature), bit i * 8 + j: visiting the set bits in order is
        // the reference's i-major loop, and every lane takes its k-th pair
        // in the same iteration
        {
            uint32_t s1[8], used1 = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int2 mj = M1[j];
                s1[j] = (uint32_t)mj.x;
                used1 |= packed_used((uint32_t)mj.y) << j;
            }
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int2 mi = M0[i];
                if (!packed_used((uint32_t)mi.y)) continue;
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (((used1 >> j) & 1u) && popc32((uint32_t)mi.x | s1[j]) <= 4)
                        pairs |= 1ull << (i * 8 + j);
            }
        }
    }
    // every lane runs the warp's largest number of admissible pairs, in step;
    // `continue` in the do-while below ends the lane's current pair
    const int rounds = __reduce_max_sync(0xffffffffu, (unsigned)popc64(pairs));
    for (int t = 0; t < rounds; t++) {
        if (pairs) {
            const int p = __ffsll((long long)pairs) - 1;
            pairs &= pairs - 1;
            const int i = p >> 3, j = p & 7;
            do {
                RCut a, b;
                load_rcut(A, (int64_t)u0 * 8 + i, M0[i], a);
                load_rcut(A, (int64_t)u1 * 8 + j, M1[j], b);
                // FindCut: first unused slot, else lowest value among
                // >2-leaf, then 2-leaf, then smaller cuts (rewrite.cu:84-109)
                int id = -1;
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (id < 0 && !sl_used(S[k])) id = k;
                if (id < 0) {
                    uint32_t best = 0xFFFFFFFFu;
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        uint32_t n = sl_n(S[k]);
                        uint32_t cls = n > 2 ? 0u : (n == 2 ? 1u : 2u);
                        uint32_t key = (cls << 20) | (sl_value(S[k]) << 3) | (uint32_t)k;
                        best = key < best ? key : best;
                    }
                    id = (int)(best & 7u);
                }
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (k == id) sl_clear_used(S[k]);
                RCut m;
                int pa, pb;
                if (!rc_merge(a, b, m, pa, pb)) continue;
                if (filter_slots(S, id, m.l, m.n, m.sign)) continue;  // dropped: slot stays free
                m.tt = rc_truth(a, b, c0, c1, pa, pb);
                const bool mini = rc_minimize(m);
                m.value = 0;
                Cut pc;
                pc.tt = m.tt;
                pc.nLeaves = m.n;
                pc.used = 1;
                pc.value = 0;
                uint32_t a0, a1;
                rc_pack_aux(m, a0, a1);
                A.cutA[q * 8 + id] = make_int2((int)a0, (int)a1);
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (k == id) {
                        S[k].l[0] = m.l[0];
                        S[k].l[1] = m.l[1];
                        S[k].l[2] = m.l[2];
                        S[k].l[3] = m.l[3];
                        S[k].sign = m.sign;
                        S[k].pk = cut_pack(pc);
                    }
                bool keep = true;
                if (mini) keep = !filter_slots(S, id, m.l, m.n, m.sign);
                pc.value = rc_value(m);
                pc.used = keep ? 1u : 0u;
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (k == id) S[k].pk = cut_pack(pc);
                if (m.n < 2) pairs = 0;  // enumeration of this node stops (rewrite.cu:291)
            } while (false);
        }
        __syncwarp();
    }
    if (!valid) return;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        A.cutL[q * 8 + k] = make_int4(S[k].l[0], S[k].l[1], S[k].l[2], S[k].l[3]);
        A.cutM[q * 8 + k] = make_int2((int)S[k].sign, (int)S[k].pk);
    }
    st_release(&A.done[q], 1);
}

// A run of wide levels, each node on one thread (throughput): the levels are
// cut into 32-node chunks that never cross a level, which warps claim in
// level order, so every fanin of a claimed node lies in an earlier, claimed
// chunk or below the run.
__global__ void __launch_bounds__(kEnumBlock, 4) k_enumerate(EnumArgs A) {
    const unsigned F = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int total = A.chunkStart[A.nLevels];
    while (true) {
        int c = 0;
        if (lane == 0) c = atomicAdd(A.counter, 1);
        c = __shfl_sync(F, c, 0);
        if (c >= total) break;
        int lo = 0, hi = A.nLevels - 1;
        while (lo < hi) {  // last level whose first chunk is <= c
            const int mid = (lo + hi + 1) >> 1;
            if (A.chunkStart[mid] <= c)
                lo = mid;
            else
                hi = mid - 1;
        }
        const int64_t q = (int64_t)A.lvlStart[lo] + (int64_t)(c - A.chunkStart[lo]) * 32 + lane;
        enum_node_thread(A, q, q < A.lvlStart[lo + 1]);
    }
}

// A run of narrower levels, each node on a warp (latency: a level's time is
// that of its slowest node), claimed in W order.  A kernel of its own for its
// smaller register need: eight resident blocks an SM instead of the four of
// one kernel for both forms (1M-AND layered graph, 3,800 nodes a level: 1.56
// ms, with six 1.64, with four 2.3).
//
// Where the forms meet (Tune::enumWideMin): a wide level takes about 30 us
// however few nodes it has, one warp's 32 replays; a warp per node takes 1.7
// ns a node and 7 us at least.  128 graphs of up to 100k ANDs: 4.3 ms with the
// line at 16,384 nodes a level, 3.77 at 32,768, 3.80 at 65,536 and 4.1 with no
// wide levels; 256 graphs of up to 200k: 12.9 at 16,384, 12.8, 14.7, 15.9.
__global__ void __launch_bounds__(kEnumBlock, 8) k_enumerate_warp(EnumArgs A) {
    __shared__ WarpCands s_cand[kEnumBlock / 32];
    const int lane = threadIdx.x & 31;
    while (true) {
        int c = 0;
        if (lane == 0) c = atomicAdd(A.counter, 1);
        c = __shfl_sync(0xffffffffu, c, 0);
        if (c >= A.q1 - A.q0) break;
        enum_node_warp(A, A.q0 + c, lane, s_cand[threadIdx.x >> 5]);
    }
}

// Runs of levels that take the same form.  Every run is a launch, which waits
// for the one before it: a profile that changes too often takes the form of
// most of its nodes throughout.
struct EnumRun {
    bool wide;
    int l0, l1;  // levels [l0, l1)
};

std::vector<EnumRun> enum_runs(const std::vector<int> &cnt, int wideMin) {
    constexpr size_t kMaxRuns = 8;
    std::vector<EnumRun> runs;
    int64_t wide = 0, all = 0;
    for (int l = 1; l < (int)cnt.size(); l++) {
        const bool w = cnt[l] >= wideMin;
        all += cnt[l];
        if (w) wide += cnt[l];
        if (runs.empty() || runs.back().wide != w)
            runs.push_back(EnumRun{w, l, l + 1});
        else
            runs.back().l1 = l + 1;
    }
    if (runs.size() > kMaxRuns) runs = {EnumRun{2 * wide > all, 1, (int)cnt.size()}};
    return runs;
}

}  // namespace

int rw_enumerate(ExecCtx &X, RwWork &w) {
    const int64_t N = w.N;
    cudaStream_t s = X.s;
    w.cutL = X.ar->get<int4>(N * 8);
    w.cutM = X.ar->get<int2>(N * 8);
    w.cutA = X.ar->get<int2>(N * 8);
    int *done = X.ar->get<int>(N);
    unsigned long long *warpPairs = reinterpret_cast<unsigned long long *>(X.counters + kCtPairs);
    if (!w.cutL || !w.cutM || !w.cutA || !done)
        return X.fail(CULS_E_OOM, "rw: scratch arena exhausted (cuts)");
    int rc;
    if ((rc = X.check(cudaMemsetAsync(w.cutM, 0, sizeof(int2) * N * 8, s), "memset"))) return rc;
    if ((rc = X.check(cudaMemsetAsync(warpPairs, 0, sizeof(unsigned long long), s), "memset"))) return rc;
    const std::vector<EnumRun> runs = enum_runs(w.lvlCnt, X.tune->enumWideMin);
    // per run: its claim counter and, if wide, its levels' starts and chunks
    const int nRuns = (int)runs.size();
    std::vector<int> host(nRuns, 0);
    std::vector<int64_t> lvlStart(w.lvlCnt.size() + 1, w.nL0);  // W position of each level's first AND node
    for (size_t l = 1; l < w.lvlCnt.size(); l++) lvlStart[l + 1] = lvlStart[l] + w.lvlCnt[l];
    for (const EnumRun &r : runs) {
        if (!r.wide) continue;
        for (int l = r.l0; l <= r.l1; l++) host.push_back((int)lvlStart[l]);
        int chunks = 0;
        for (int l = r.l0; l <= r.l1; l++) {
            host.push_back(chunks);
            if (l < r.l1) chunks += (w.lvlCnt[l] + 31) / 32;
        }
    }
    int *dev = X.ar->get<int>(host.size() + 1);
    if (!dev) return X.fail(CULS_E_OOM, "rw: scratch arena exhausted (levels)");
    if (nRuns && (rc = X.check(cudaMemcpyAsync(dev, host.data(), sizeof(int) * host.size(), cudaMemcpyHostToDevice, s), "h2d")))
        return rc;
    k_enum_init<<<X.grid(N), kBlock, 0, s>>>(N, w.wlev, w.wl, w.lidLow, w.ref, w.cutL, w.cutM, w.cutA, done);
    X.launched(1);
    X.mark(kMkEnumK0);
    const int *table = dev + nRuns;
    for (int k = 0; k < nRuns; k++) {
        const EnumRun &r = runs[k];
        const int n = r.l1 - r.l0;
        EnumArgs A{lvlStart[r.l0], lvlStart[r.l1], n,        table,    table + n + 1, w.w0, w.w1, w.ref,
                   w.lidLow,       w.cutL,         w.cutM,   w.cutA,   done,          dev + k, warpPairs, X.status};
        const int64_t width = (A.q1 - A.q0) / n + 1;
        // a wide run fills the GPU; a narrow one runs about sixteen levels'
        // worth of nodes at a time
        if (r.wide) {
            table += 2 * (n + 1);
            k_enumerate<<<flow_blocks(width, kEnumBlock, (unsigned)(X.sms * X.tune->enumBlocksPerSm), X.sms), kEnumBlock, 0,
                          s>>>(A);
        } else {
            k_enumerate_warp<<<flow_blocks(width, kEnumBlock / 32, (unsigned)(X.sms * std::min(X.tune->enumBlocksPerSm, 8)),
                                           X.sms), kEnumBlock, 0, s>>>(A);
        }
        X.launched(1);
    }
    X.mark(kMkEnumK1);
    if ((rc = X.check(cudaGetLastError(), "enumerate launch"))) return rc;
    return 0;
}

}  // namespace culs
