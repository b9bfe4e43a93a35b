// Register-resident cut enumeration for one node (device side of
// k_enumerate).  Same semantics as enum_pair()/CutEnumerate
// (src/algorithms/rewrite.cu:268-294): the 8 slots live in registers (every
// slot index is a compile-time constant after unrolling), and every cut
// carries, beside its leaves, each leaf's reference count (clamped to 1001)
// and local-id bits, so cut values and minimised signatures need no memory
// access.
#pragma once

#include "rw_core.cuh"

namespace culs {

// A cut in registers.  Each leaf's attributes, its reference count (11 bits)
// and local-id bits (5), are a halfword: aux0 = leaves 0 and 1, aux1 = leaves
// 2 and 3.  Refs are clamped to 1001, which leaves CutFindValue's result
// unchanged (it caps the sum at 1000).  Unused places hold zeros.
struct RCut {
    int l[4];
    uint32_t sign, tt, value, n, used;
    uint32_t ref[4];
    uint32_t lid[4];
};

__device__ __forceinline__ uint32_t rc_attr(const RCut &c, int i) { return (c.ref[i] & 0x7FFu) | ((c.lid[i] & 31u) << 11); }
__device__ __forceinline__ void rc_set_attr(RCut &c, int i, uint32_t a) {
    c.ref[i] = a & 0x7FFu;
    c.lid[i] = (a >> 11) & 31u;
}

__device__ __forceinline__ void rc_unpack_aux(uint32_t a0, uint32_t a1, RCut &c) {
    rc_set_attr(c, 0, a0 & 0xFFFFu);
    rc_set_attr(c, 1, a0 >> 16);
    rc_set_attr(c, 2, a1 & 0xFFFFu);
    rc_set_attr(c, 3, a1 >> 16);
}

__device__ __forceinline__ void rc_pack_aux(const RCut &c, uint32_t &a0, uint32_t &a1) {
    a0 = rc_attr(c, 0) | (rc_attr(c, 1) << 16);
    a1 = rc_attr(c, 2) | (rc_attr(c, 3) << 16);
}

// CutFindValue from the carried refs.
__device__ __forceinline__ uint32_t rc_value(const RCut &c) {
    if (c.n < 2) return 1001u;
    const uint32_t v = c.ref[0] + c.ref[1] + c.ref[2] + c.ref[3];
    const uint32_t ones = (c.ref[0] == 1u) + (c.ref[1] == 1u) + (c.ref[2] == 1u) + (c.ref[3] == 1u);
    int value = v > 1000u ? 1000 : (int)v;
    if (ones > 3) value = 5 - (int)ones;
    return (uint32_t)value & 0x7FFu;
}

// MergeCutOrdered / MergeCut with the leaf attributes carried along: four
// merge steps, each taking the smaller head leaf (both when equal) and moving
// the lists up, without branches -- the lanes of the warp-wide enumeration
// merge different cuts.  Places past a list's end are larger than every leaf.
// Bit s of pa (pb) is set when a (b) has the merged leaf s: CutTruthPhase
// (rewrite.cu:195-201).
__device__ __forceinline__ bool rc_merge(const RCut &a, const RCut &b, RCut &o, int &pa, int &pb) {
    constexpr int kEnd = 0x7FFFFFFF;
    int x[4], y[4];
    uint32_t xa[4], ya[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        x[i] = (uint32_t)i < a.n ? a.l[i] : kEnd;
        y[i] = (uint32_t)i < b.n ? b.l[i] : kEnd;
        xa[i] = rc_attr(a, i);
        ya[i] = rc_attr(b, i);
    }
    const bool first = a.n >= b.n;  // whose attributes an equal leaf takes
    int c = 0;
    pa = pb = 0;
#pragma unroll
    for (int s = 0; s < 4; s++) {
        const bool ta = x[0] <= y[0], tb = y[0] <= x[0];
        const int leaf = ta ? x[0] : y[0];
        const bool act = leaf != kEnd;
        o.l[s] = act ? leaf : 0;
        rc_set_attr(o, s, act ? (ta && (first || !tb) ? xa[0] : ya[0]) : 0u);
        pa |= act && ta ? 1 << s : 0;
        pb |= act && tb ? 1 << s : 0;
        c += act ? 1 : 0;
        // what is still looked at: the heads of the steps left, and the last
        // one's successor
#pragma unroll
        for (int i = 0; i < 4 - s; i++) {
            x[i] = ta ? (i < 3 ? x[i + 1] : kEnd) : x[i];
            y[i] = tb ? (i < 3 ? y[i + 1] : kEnd) : y[i];
            if (i < 3 - s) {
                xa[i] = ta && i < 3 ? xa[i + 1] : xa[i];
                ya[i] = tb && i < 3 ? ya[i + 1] : ya[i];
            }
        }
    }
    o.n = (uint32_t)c;
    o.sign = a.sign | b.sign;
    o.used = 1;
    return x[0] == kEnd && y[0] == kEnd;
}

// CutTruthtable (rewrite.cu:223-229); pa, pb as rc_merge gives them.
__device__ __forceinline__ uint32_t rc_truth(const RCut &a, const RCut &b, int ca, int cb, int pa, int pb) {
    uint32_t t0 = ca ? (~a.tt & 0xFFFFu) : a.tt;
    uint32_t t1 = cb ? (~b.tt & 0xFFFFu) : b.tt;
    t0 = tt_stretch_flat(t0, (int)a.n, pa);
    t1 = tt_stretch_flat(t1, (int)b.n, pb);
    return (t0 & t1) & 0xFFFFu;
}

// MinimizeCutSupport with carried attributes; returns true when leaves were
// removed.
__device__ __forceinline__ bool rc_minimize(RCut &c) {
    const uint32_t m0[4] = {0x5555u, 0x3333u, 0x0F0Fu, 0x00FFu};
    const uint32_t m1[4] = {0xAAAAu, 0xCCCCu, 0xF0F0u, 0xFF00u};
    int ph = 0, nl = (int)c.n;
    const uint32_t t = c.tt & 0xFFFFu;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if ((uint32_t)i >= c.n) continue;
        if ((t & m0[i]) == ((t & m1[i]) >> (1 << i)))
            nl--;
        else
            ph |= 1 << i;
    }
    if (nl == (int)c.n) return false;
    c.tt = tt_shrink_flat(t, ph) & 0xFFFFu;
    RCut o = c;
#pragma unroll
    for (int s = 0; s < 4; s++) {
        o.l[s] = 0;
        rc_set_attr(o, s, 0);
    }
    int k = 0;
    uint32_t sign = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if ((uint32_t)i < c.n && (ph >> i & 1)) {
            // k <= i, so writing slot k never clobbers an unread slot
#pragma unroll
            for (int s = 0; s < 4; s++)
                if (s == k) {
                    o.l[s] = c.l[i];
                    rc_set_attr(o, s, rc_attr(c, i));
                }
            sign |= 1u << c.lid[i];
            k++;
        }
    }
    o.sign = sign;
    o.n = (uint32_t)nl;
    c = o;
    return true;
}

}  // namespace culs
