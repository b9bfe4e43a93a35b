// Per-item logic of the rewriting pass, written as __host__ __device__
// functions over plain arrays.  The engine's kernels (engine.cu) call these;
// each function names the reference code whose semantics it reproduces
// (paths relative to the CULS source tree).
//
// Node addressing: every object of a batch has a storage position; literals
// are 2*position + complement.  Within one graph, storage order equals id
// order, so comparisons of positions reproduce the reference's comparisons of
// node ids.  Per graph, `cpos` is the position of the constant node.
#pragma once

#include "common.cuh"
#ifdef __CUDACC__
#include "prim.cuh"
#endif

namespace culs {

// ----------------------------------------------------------- library
// The 4-input rewriting library (same values as CULS
// src/algorithms/rewrite_library.inc, decoded as rw::CPUSolver::ReadLibrary
// does, src/algorithms/rewrite.cu:1281-1307), repacked for single loads.
constexpr int kNumClasses = 222;
constexpr int kMaxLibNodes = 56;  // <= 50 internal nodes + 4 inputs fit in 54
struct RwLib {
    // per truth table: phase (bits 0-4) | perm index (bits 8-12) | class (bits 16-23)
    uint32_t npn[1 << 16];
    uint8_t perm4[24][4];
    uint8_t nNodes[kNumClasses], nRoots[kNumClasses];
    // per class and internal node j (library index j+4):
    // fanin0 (bits 0-7) | fanin1 (bits 8-15) | compl0 (bit 16) | compl1 (bit 17)
    uint32_t node[kNumClasses][kMaxLibNodes];
    uint8_t roots[kNumClasses][16];
    // Evaluation reaches a library node through a matched fanin, or, when
    // both its fanins are inputs, through the pair's filter bits:
    // uses[j]: the nodes that read node j;
    // pairNode[4 * pair + 2 * c_lo + c_hi]: the node that ANDs inputs lo < hi
    // with these complements, pairs in the order 01 02 03 12 13 23, 0 when
    // there is none, and pairMask its non-zero entries;
    // pairRest: nodes over two inputs that have no entry of their own.
    unsigned long long uses[kNumClasses][kMaxLibNodes];
    uint8_t pairNode[kNumClasses][24];
    uint32_t pairMask[kNumClasses];
    unsigned long long pairRest[kNumClasses];
    // Per class and root: the pair entries in its cone (bits 0-23), and bit 31
    // when the root itself is not one of them.
    uint32_t rootPairs[kNumClasses][16];
    // Per class and root: bit j set for every internal node j (j >= 4) in
    // the root's cone, the root included.
    unsigned long long rootCone[kNumClasses][16];
    // Per class and root: byte i = 1 + the longest path from input i to the
    // root, 0 when the root does not depend on it.
    uint32_t rootDepth[kNumClasses][16];
};

CULS_HD int npn_phase(uint32_t w) { return (int)(w & 31u); }
CULS_HD int npn_perm(uint32_t w) { return (int)((w >> 8) & 31u); }
CULS_HD int npn_class(uint32_t w) { return (int)((w >> 16) & 255u); }
CULS_HD int ln_f0(uint32_t w) { return (int)(w & 255u); }
CULS_HD int ln_f1(uint32_t w) { return (int)((w >> 8) & 255u); }
CULS_HD int ln_c0(uint32_t w) { return (int)((w >> 16) & 1u); }
CULS_HD int ln_c1(uint32_t w) { return (int)((w >> 17) & 1u); }

// --------------------------------------------------------------- cuts
// A cut slot (rw::Cut, src/algorithms/rewrite.h:10-16).  In device memory a
// slot is an int4 of leaves plus an int2 {sign, packed}, packed =
// tt (bits 0-15) | value (bits 16-26) | nLeaves (bits 27-29) | used (bit 30).
struct Cut {
    int leaves[4];
    uint32_t sign;
    uint32_t tt;
    uint32_t value;
    uint32_t nLeaves;
    uint32_t used;
};

CULS_HD uint32_t cut_pack(const Cut &c) {
    return (c.tt & 0xFFFFu) | ((c.value & 0x7FFu) << 16) | ((c.nLeaves & 7u) << 27) | ((c.used & 1u) << 30);
}
CULS_HD void cut_unpack(uint32_t w, Cut &c) {
    c.tt = w & 0xFFFFu;
    c.value = (w >> 16) & 0x7FFu;
    c.nLeaves = (w >> 27) & 7u;
    c.used = (w >> 30) & 1u;
}
CULS_HD uint32_t packed_used(uint32_t w) { return (w >> 30) & 1u; }
CULS_HD uint32_t packed_nleaves(uint32_t w) { return (w >> 27) & 7u; }

CULS_HD int popc32(uint32_t x) {
#if defined(__CUDA_ARCH__)
    return __popc(x);
#else
    return __builtin_popcount(x);
#endif
}
CULS_HD int popc64(uint64_t x) {
#if defined(__CUDA_ARCH__)
    return __popcll(x);
#else
    return __builtin_popcountll(x);
#endif
}

// CutFindValue, src/algorithms/rewrite.cu:49-61
CULS_HD uint32_t cut_value(const Cut &c, const int *ref) {
    int value = 0, nOnes = 0;
    for (uint32_t i = 0; i < c.nLeaves; i++) {
        int r = ref[c.leaves[i]];
        value += r;
        nOnes += (r == 1);
    }
    if (c.nLeaves < 2) return 1001u;
    if (value > 1000) value = 1000;
    if (nOnes > 3) value = 5 - nOnes;
    return (uint32_t)value & 0x7FFu;
}

// FindCut, src/algorithms/rewrite.cu:84-109: first unused slot, else the
// lowest-value slot among >2-leaf cuts, then 2-leaf, then smaller cuts; the
// chosen slot is marked unused before any merge is tried.
CULS_HD int find_slot(Cut *s) {
    for (int i = 0; i < 8; i++)
        if (s[i].used == 0) return i;
    int ans = -1;
    for (int i = 0; i < 8; i++)
        if (s[i].nLeaves > 2 && (ans == -1 || s[i].value < s[ans].value)) ans = i;
    if (ans == -1)
        for (int i = 0; i < 8; i++)
            if (s[i].nLeaves == 2 && (ans == -1 || s[i].value < s[ans].value)) ans = i;
    if (ans == -1)
        for (int i = 0; i < 8; i++)
            if (s[i].nLeaves < 2 && (ans == -1 || s[i].value < s[ans].value)) ans = i;
    s[ans].used = 0;
    return ans;
}

// MergeCutOrdered / MergeCut, src/algorithms/rewrite.cu:112-164.  Merges
// the sorted leaf lists of a and b into out (at most 4 leaves).  Returns 0
// when the union exceeds 4 leaves; out's leaves may be partly written then.
CULS_HD int merge_cuts(const Cut &a0, const Cut &b0, Cut *out) {
    const Cut &a = (a0.nLeaves >= b0.nLeaves) ? a0 : b0;
    const Cut &b = (a0.nLeaves >= b0.nLeaves) ? b0 : a0;
    int c = 0, i = 0, k = 0;
    const int na = (int)a.nLeaves, nb = (int)b.nLeaves;
    for (c = 0; c < 4; c++) {
        if (k == nb) {
            if (i == na) {
                out->nLeaves = (uint32_t)c;
                out->sign = a0.sign | b0.sign;
                out->used = 1;
                return 1;
            }
            out->leaves[c] = a.leaves[i++];
            continue;
        }
        if (i == na) {
            out->leaves[c] = b.leaves[k++];
            continue;
        }
        if (a.leaves[i] < b.leaves[k]) {
            out->leaves[c] = a.leaves[i++];
            continue;
        }
        if (a.leaves[i] > b.leaves[k]) {
            out->leaves[c] = b.leaves[k++];
            continue;
        }
        out->leaves[c] = a.leaves[i++];
        k++;
    }
    if (i < na || k < nb) return 0;
    out->nLeaves = (uint32_t)c;
    out->sign = a0.sign | b0.sign;
    out->used = 1;
    return 1;
}

// CutDominance, src/algorithms/rewrite.cu:167-175: leaves(a) subset of leaves(b)
CULS_HD int cut_subset(const Cut &a, const Cut &b) {
    for (uint32_t i = 0; i < a.nLeaves; i++) {
        int ok = 0;
        for (uint32_t j = 0; j < b.nLeaves; j++)
            if (b.leaves[j] == a.leaves[i]) ok = 1;
        if (!ok) return 0;
    }
    return 1;
}

// CutFilter, src/algorithms/rewrite.cu:178-193
CULS_HD int cut_filter(Cut *s, int id) {
    for (int i = 0; i < 8; i++) {
        if (i == id || !s[i].used) continue;
        if (s[i].nLeaves > s[id].nLeaves) {
            if ((s[i].sign & s[id].sign) != s[id].sign) continue;
            if (cut_subset(s[id], s[i])) s[i].used = 0;
        } else {
            if ((s[i].sign & s[id].sign) != s[i].sign) continue;
            if (cut_subset(s[i], s[id])) {
                s[id].used = 0;
                return 1;
            }
        }
    }
    return 0;
}

// CutTruthSwapAdjacentVars, src/algorithms/rewrite.cu:203-211, on 16 bits.
CULS_HD uint32_t tt_swap_adj(uint32_t t, int v) {
    if (v == 0) return (t & 0x9999u) | ((t & 0x2222u) << 1) | ((t & 0x4444u) >> 1);
    if (v == 1) return (t & 0xC3C3u) | ((t & 0x0C0Cu) << 2) | ((t & 0x3030u) >> 2);
    if (v == 2) return (t & 0xF00Fu) | ((t & 0x00F0u) << 4) | ((t & 0x0F00u) >> 4);
    return 0;
}

// CutTruthPhase, src/algorithms/rewrite.cu:195-201
CULS_HD int tt_phase(const Cut &x, const Cut &cut) {
    int ph = 0;
    for (uint32_t i = 0; i < cut.nLeaves; i++)
        for (uint32_t j = 0; j < x.nLeaves; j++)
            if (x.leaves[j] == cut.leaves[i]) ph |= 1 << i;
    return ph;
}

// CutTruthStretch, src/algorithms/rewrite.cu:213-221
CULS_HD uint32_t tt_stretch(uint32_t t, int nVar, int ph) {
    int var = nVar - 1;
    for (int i = 3; i >= 0; i--)
        if (ph >> i & 1) {
            for (int k = var; k < i; k++) t = tt_swap_adj(t, k);
            var--;
        }
    return t;
}

// tt_swap_adj with the variable known at compile time
template <int V>
CULS_HD uint32_t tt_swap_adj_c(uint32_t t) {
    return V == 0   ? (t & 0x9999u) | ((t & 0x2222u) << 1) | ((t & 0x4444u) >> 1)
           : V == 1 ? (t & 0xC3C3u) | ((t & 0x0C0Cu) << 2) | ((t & 0x3030u) >> 2)
                    : (t & 0xF00Fu) | ((t & 0x00F0u) << 4) | ((t & 0x0F00u) >> 4);
}

// tt_stretch without branches, for the warp-wide enumeration (lanes with
// different phases take one path): every swap the loops could make, in the
// loops' order, applied when the loops would make it.  Equal to tt_stretch
// whenever ph has nVar bits set, which holds for every call (a fanin cut's
// leaves all appear in the merged cut).
CULS_HD uint32_t tt_stretch_flat(uint32_t t, int nVar, int ph) {
    int var = nVar - 1;
#define CULS_SW(K, I)                                                          \
    {                                                                          \
        const uint32_t sw = tt_swap_adj_c<K>(t);                               \
        t = (((ph >> (I)) & 1) && (K) >= var) ? sw : t;                        \
    }
    CULS_SW(0, 3) CULS_SW(1, 3) CULS_SW(2, 3) var -= (ph >> 3) & 1;
    CULS_SW(0, 2) CULS_SW(1, 2) var -= (ph >> 2) & 1;
    CULS_SW(0, 1)
#undef CULS_SW
    return t;
}

// CutTruthtable, src/algorithms/rewrite.cu:223-229
CULS_HD uint32_t cut_truth(const Cut &cut, const Cut &a, const Cut &b, int ca, int cb) {
    uint32_t t0 = ca ? (~a.tt & 0xFFFFu) : a.tt;
    uint32_t t1 = cb ? (~b.tt & 0xFFFFu) : b.tt;
    t0 = tt_stretch(t0, (int)a.nLeaves, tt_phase(a, cut));
    t1 = tt_stretch(t1, (int)b.nLeaves, tt_phase(b, cut));
    return (t0 & t1) & 0xFFFFu;
}

// CutTruthShrink, src/algorithms/rewrite.cu:231-241
CULS_HD uint32_t tt_shrink(uint32_t t, int ph) {
    int var = 0;
    for (int i = 0; i < 4; i++)
        if (ph & (1 << i)) {
            for (int k = i - 1; k >= var; k--) t = tt_swap_adj(t, k);
            var++;
        }
    return t;
}

// tt_shrink without branches (see tt_stretch_flat): equal to tt_shrink for
// every phase.
CULS_HD uint32_t tt_shrink_flat(uint32_t t, int ph) {
    int var = (ph & 1);
#define CULS_SW(K, I)                                                          \
    {                                                                          \
        const uint32_t sw = tt_swap_adj_c<K>(t);                               \
        t = (((ph >> (I)) & 1) && (K) >= var) ? sw : t;                        \
    }
    CULS_SW(0, 1) var += (ph >> 1) & 1;
    CULS_SW(1, 2) CULS_SW(0, 2) var += (ph >> 2) & 1;
    CULS_SW(2, 3) CULS_SW(1, 3) CULS_SW(0, 3)
#undef CULS_SW
    return t;
}

// MinimizeCutSupport, src/algorithms/rewrite.cu:243-266.  `lsb` holds
// (local id & 31) of each leaf position so that the recomputed sign uses
// graph-local ids; it is read through lidLow[leaf].
CULS_HD int cut_minimize(Cut *c, const uint8_t *lidLow) {
    const uint32_t m0[4] = {0x5555u, 0x3333u, 0x0F0Fu, 0x00FFu};
    const uint32_t m1[4] = {0xAAAAu, 0xCCCCu, 0xF0F0u, 0xFF00u};
    int ph = 0;
    uint32_t t = c->tt & 0xFFFFu;
    int nl = (int)c->nLeaves;
    for (uint32_t i = 0; i < c->nLeaves; i++) {
        if ((t & m0[i]) == ((t & m1[i]) >> (1 << i)))
            nl--;
        else
            ph |= 1 << i;
    }
    if (nl == (int)c->nLeaves) return 0;
    t = tt_shrink(t, ph);
    c->tt = t & 0xFFFFu;
    c->sign = 0;
    for (uint32_t i = 0, k = 0; i < c->nLeaves; i++)
        if (ph >> i & 1) {
            c->leaves[k++] = c->leaves[i];
            c->sign |= 1u << (lidLow[c->leaves[i]] & 31u);
        }
    c->nLeaves = (uint32_t)nl;
    return 1;
}

// The CutEnumerate body for one pair (src/algorithms/rewrite.cu:282-291).
// Returns 1 when enumeration of this node must stop (a cut with fewer than
// two leaves was produced).
CULS_HD int enum_pair(Cut *s, const Cut &a, const Cut &b, int ca, int cb, const int *ref, const uint8_t *lidLow) {
    if (popc32(a.sign | b.sign) > 4) return 0;
    int id = find_slot(s);
    if (!merge_cuts(a, b, &s[id])) return 0;
    if (cut_filter(s, id)) return 0;
    s[id].tt = cut_truth(s[id], a, b, ca, cb);
    if (cut_minimize(&s[id], lidLow)) cut_filter(s, id);
    s[id].value = cut_value(s[id], ref);
    return s[id].nLeaves < 2 ? 1 : 0;
}

// ------------------------------------------------------ existence table
// Open-addressing table of AND nodes keyed by (fanin0 id, fanin1 id,
// compl0, compl1): the role of BuildHashTable/TableLookup
// (src/algorithms/rewrite.cu:328-367,450-471).  Duplicate keys keep the
// smallest position.
CULS_HD unsigned long long and_key(int in0, int in1, int c0, int c1) {
    return ((unsigned long long)(uint32_t)in0 << 32) | ((unsigned long long)(uint32_t)in1 << 2) |
           ((unsigned long long)c0 << 1) | (unsigned long long)c1;
}

// A slot holds its key and, in one 64-bit word, the lowest rank inserted
// with it and that insertion's position (rank << 32 | position), so that an
// insertion's CAS and min touch one 32-byte sector and a lookup finds the
// winner's position without a rank-to-position table.  Empty: key
// kEmptyKey, rank and position kEmptyRp.
struct alignas(16) AndSlot {
    unsigned long long key;
    unsigned long long rp;
};
constexpr unsigned long long kEmptyRp = 0x7F7F7F7F7F7F7F7Full;
CULS_HD int slot_rank(unsigned long long rp) { return (int)(rp >> 32); }
CULS_HD int slot_pos(unsigned long long rp) { return (int)(uint32_t)rp; }

struct AndTable {
    AndSlot *slots;
    uint32_t mask;  // capacity - 1 (capacity is a power of two)
};

#ifdef __CUDACC__
// Empties n slots on stream s.
inline cudaError_t and_table_clear(AndSlot *slots, int64_t n, cudaStream_t s) {
    return fill_i4(reinterpret_cast<int4 *>(slots), make_int4(-1, -1, 0x7F7F7F7F, 0x7F7F7F7F), n, s);
}
#endif

// Inserts key with (rank, pos): the slot keeps the lowest rank and its
// position.  Returns the slot, or -1 (and kDevTableFull) when the probe
// sequence runs out.
CULS_HD int table_insert(const AndTable &t, unsigned long long key, int rank, int pos, int *status) {
    uint32_t h = (uint32_t)mix64(key) & t.mask;
    for (uint32_t probe = 0; probe <= t.mask; probe++) {
        unsigned long long prev = at_cas(&t.slots[h].key, kEmptyKey, key);
        if (prev == kEmptyKey || prev == key) {
            at_min(&t.slots[h].rp, ((unsigned long long)(uint32_t)rank << 32) | (uint32_t)pos);
            return (int)h;
        }
        h = (h + 1) & t.mask;
    }
    set_status(status, kDevTableFull);
    return -1;
}

// Returns the lowest rank stored for key, or -1 when absent.
CULS_HD int table_find(const AndTable &t, unsigned long long key, int *status) {
    uint32_t h = (uint32_t)mix64(key) & t.mask;
    for (uint32_t probe = 0; probe <= t.mask; probe++) {
        unsigned long long k = t.slots[h].key;
        if (k == key) return slot_rank(t.slots[h].rp);
        if (k == kEmptyKey) return -1;
        h = (h + 1) & t.mask;
    }
    set_status(status, kDevTableFull);
    return -1;
}

// TableLookup, src/algorithms/rewrite.cu:346-367 (ids swapped, not literals)
CULS_HD int and_lookup(const AndTable &t, int in0, int in1, int c0, int c1, int *status) {
    if (in0 > in1) {
        int x = in0;
        in0 = in1;
        in1 = x;
        x = c0;
        c0 = c1;
        c1 = x;
    }
    return table_find(t, and_key(in0, in1, c0, c1), status);
}

// ---------------------------------------- per-graph existence table
// The existence table of one rewriting pass, split by graph: graph g owns
// slots [off[g], off[g + 1]) and only its own nodes are inserted into or
// looked up in that region, so passes that visit the nodes graph by graph
// keep the region they probe resident in L2.  A slot is 16 bytes {key,
// value}, so a probe touches one sector.  Duplicate keys keep the smallest
// position, as in AndTable.
struct alignas(16) TabSlot {
    unsigned long long key;
    int val;  // smallest position with this key
    int pad;
};

struct RegionTable {
    TabSlot *slots;
    const int64_t *off;  // G + 1 slot offsets
};

struct TabRegion {
    TabSlot *slots;
    uint32_t size;
};

CULS_HD TabRegion table_region(const RegionTable &t, int g) {
    const int64_t a = t.off[g], b = t.off[g + 1];
    return TabRegion{t.slots + a, (uint32_t)(b - a)};
}

// Home slot: a multiplicative hash of the key's two 32-bit halves (odd
// constants from the golden ratio and MurmurHash3), its high bits scaled
// onto [0, size) by a multiply-high.  Two 32-bit multiplies keep the probe
// short; linear probing at load <= 1/2 tolerates its weaker mixing.
CULS_HD uint32_t region_home(unsigned long long key, uint32_t size) {
    const uint32_t h = (uint32_t)(key >> 32) * 0x9E3779B1u + (uint32_t)key * 0x85EBCA6Bu;
    return (uint32_t)(((unsigned long long)(h ^ (h >> 15)) * size) >> 32);
}

CULS_HD int region_insert(const TabRegion &t, unsigned long long key, int val, int *status) {
    uint32_t h = region_home(key, t.size);
    for (uint32_t probe = 0; probe < t.size; probe++) {
        unsigned long long prev = at_cas(&t.slots[h].key, kEmptyKey, key);
        if (prev == kEmptyKey || prev == key) {
            at_min(&t.slots[h].val, val);
            return (int)h;
        }
        if (++h == t.size) h = 0;
    }
    set_status(status, kDevTableFull);
    return -1;
}

// Lookup in a region that no thread writes during the calling kernel.
CULS_HD int region_find(const TabRegion &t, unsigned long long key, int *status) {
    uint32_t h = region_home(key, t.size);
    for (uint32_t probe = 0; probe < t.size; probe++) {
#if defined(__CUDA_ARCH__)
        const int4 s = *reinterpret_cast<const int4 *>(&t.slots[h]);
        const unsigned long long k = ((unsigned long long)(uint32_t)s.y << 32) | (uint32_t)s.x;
        if (k == key) return s.z;
#else
        const unsigned long long k = t.slots[h].key;
        if (k == key) return t.slots[h].val;
#endif
        if (k == kEmptyKey) return -1;
        if (++h == t.size) h = 0;
    }
    set_status(status, kDevTableFull);
    return -1;
}

// TableLookup (src/algorithms/rewrite.cu:346-367) on a graph's region.
CULS_HD int region_and_lookup(const TabRegion &t, int in0, int in1, int c0, int c1, int *status) {
    if (in0 > in1) {
        int x = in0;
        in0 = in1;
        in1 = x;
        x = c0;
        c0 = c1;
        c1 = x;
    }
    return region_find(t, and_key(in0, in1, c0, c1), status);
}

// --------------------------------------------------------- evaluation
struct EvalIn {
    const int *L0, *L1;  // fanin literals (the constant and PIs point at the constant)
    const int *ref;      // fanout counts incl. PO references
    const int *level;
    const RwLib *lib;
    TabRegion tab;       // the region of the evaluated node's graph
    const unsigned long long *pairs;  // per node: the filter of its table keys (pair_bit)
    int *status;
};

// A node's 64-bit filter says which ANDs it may be the higher fanin of: bit
// pair_bit(lo) + 2 * c_lo + c_hi is set for every key (lo, this node, c_lo,
// c_hi) in the table.  A clear bit proves the key absent.
// Four such words a cut, read for all six input pairs, stand in for most of
// the table probes that fail.
CULS_HD int pair_bit(int lo) { return (int)(((uint32_t)lo * 0x9E3779B1u) >> 28) << 2; }

CULS_HD int ctz64(uint64_t x) {
#if defined(__CUDA_ARCH__)
    return __ffsll((long long)x) - 1;
#else
    return __builtin_ctzll(x);
#endif
}

// CalcMFFC (src/algorithms/rewrite.cu:296-326) of root: its count, and the
// nDel table entries whose reference count reached zero, which are those that
// IsDeleted reports, at del (room for 8).
//
// The reference's table of 8 entries is held as ids in registers, every access
// by a literal index, and a byte per count.  A byte is enough: at most nine
// nodes are entered, so at most 18 decrements happen, and a count that starts
// at 255 or above never reaches zero.  The recursion visits a node's first
// fanin and what is below it before the second, so the second fanins wait on a
// stack, one per node entered.
CULS_HD int mffc_size(const EvalIn &E, int root, const int (&leaves)[4], int *del, int *nDel) {
    int id[8], wait[10];
#pragma unroll
    for (int k = 0; k < 8; k++) id[k] = -1;
    uint64_t counts = 0;
    int size = 0, sp = 1, count = 1;
    wait[0] = E.L1[root] >> 1;
    int v = E.L0[root] >> 1;
    while (true) {
        bool zero = false;  // Decrease(v) returned zero
        if (v != leaves[0] && v != leaves[1] && v != leaves[2] && v != leaves[3]) {
            uint32_t at = 0;
#pragma unroll
            for (int k = 0; k < 8; k++) at |= id[k] == v ? 1u << k : 0u;
            if (at) {
                const int sh = 8 * ctz64(at);
                const uint64_t c = (counts >> sh) & 255u, c1 = (c - 1) & 255u;
                counts ^= (c ^ c1) << sh;
                zero = c1 == 0;
            } else if (size < 8) {  // a full table returns 1
                const uint32_t r = (uint32_t)E.ref[v] - 1u;
#pragma unroll
                for (int k = 0; k < 8; k++) id[k] = k == size ? v : id[k];
                counts |= (uint64_t)(r < 255u ? r : 255u) << (8 * size);
                size++;
                zero = r == 0;
            }
        }
        if (zero) {
            count++;
            wait[sp++] = E.L1[v] >> 1;
            v = E.L0[v] >> 1;
        } else {
            if (sp == 0) break;
            v = wait[--sp];
        }
    }
    int n = 0;
#pragma unroll
    for (int k = 0; k < 8; k++)
        if (k < size && ((counts >> (8 * k)) & 255u) == 0) del[n++] = id[k];
    *nDel = n;
    return count;
}

// True when CalcMFFC of root w.r.t. these leaves is the root alone and no
// table count reaches zero: its first two Decrease calls (the root's
// fanins) are then all that runs.  A count reaches zero only for a fanin that
// is not a leaf and has one reference, or -- both fanins the same node -- two.
CULS_HD bool mffc_trivial(const EvalIn &E, int root, const int (&leaves)[4]) {
    const int f0 = E.L0[root] >> 1, f1 = E.L1[root] >> 1;
    const bool l0 = f0 == leaves[0] || f0 == leaves[1] || f0 == leaves[2] || f0 == leaves[3];
    const bool l1 = f1 == leaves[0] || f1 == leaves[1] || f1 == leaves[2] || f1 == leaves[3];
    if (f0 == f1) return l0 || E.ref[f0] > 2;
    return (l0 || E.ref[f0] >= 2) && (l1 || E.ref[f1] >= 2);
}

// IsDeleted (src/algorithms/rewrite.cu:312-316) on the MFFC's nodes: the
// table entries whose count reached zero, nDel of them at del.
CULS_HD bool mffc_member(int v, int nDel, const int *del) {
    for (int j = 0; j < nDel; j++)
        if (del[j] == v) return true;
    return false;
}

// The four complement combinations of the AND of inputs lo < hi (nodes a and
// b, input complements na and nb) that the filters leave possible, as bits
// 2 * c_lo + c_hi in the library's terms.
CULS_HD uint32_t pair_possible(int a, int b, unsigned long long fa, unsigned long long fb, int na, int nb) {
    const bool sw = a > b;  // TableLookup orders the ids
    uint32_t n = (uint32_t)((sw ? fa : fb) >> pair_bit(sw ? b : a)) & 15u;
    if (!n) return 0;
    const uint32_t t = (n & 9u) | ((n & 2u) << 1) | ((n & 4u) >> 1);
    if (sw) n = t;
    if (a == b) n |= t;
    if (na) n = ((n << 2) | (n >> 2)) & 15u;
    if (nb) n = ((n & 5u) << 1) | ((n >> 1) & 5u);
    return n;
}

// A cut as its class sees it: the four inputs' nodes, their complements (the
// reference's isC mask only has input bits, 0..3), and the class's pair
// entries that the filters leave possible.
struct CutView {
    int in[4];
    int isC, cls;
    uint32_t possible;
};

CULS_HD CutView cut_view(const EvalIn &E, int cpos, uint32_t pk, int4 l) {
    CutView v;
    const uint32_t npn = E.lib->npn[pk & 0xFFFFu];
    v.isC = npn_phase(npn) & 15;
    v.cls = npn_class(npn);
    const uint32_t perm = *reinterpret_cast<const uint32_t *>(E.lib->perm4[npn_perm(npn)]);
    const int leaves[4] = {l.x, l.y, l.z, packed_nleaves(pk) == 3 ? cpos : l.w};
    unsigned long long f[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int p = (int)((perm >> (8 * j)) & 255u);
        v.in[j] = p == 0 ? leaves[0] : (p == 1 ? leaves[1] : (p == 2 ? leaves[2] : leaves[3]));
        f[j] = E.pairs[v.in[j]];
    }
    v.possible = 0;
#pragma unroll
    for (int i = 0, k = 0; i < 3; i++)
#pragma unroll
        for (int j = i + 1; j < 4; j++, k += 4)
            v.possible |= pair_possible(v.in[i], v.in[j], f[i], f[j], (v.isC >> i) & 1, (v.isC >> j) & 1) << k;
    v.possible &= E.lib->pairMask[v.cls];
    return v;
}

// The roots that may add no more than spare nodes, as a mask: a cone's pair
// nodes that are not possible stay unmatched, and with them the root above
// them.  Most cuts are left with one or two roots, one of them the node's own
// structure.
CULS_HD uint32_t open_roots(const EvalIn &E, const CutView &v, int spare) {
    const int nr = E.lib->nRoots[v.cls];
    uint32_t open = 0;
    for (int out = 0; out < nr; out++) {
        const uint32_t p = E.lib->rootPairs[v.cls][out];
        const int missing = popc32(p & 0xFFFFFFu & ~v.possible);
        if (missing + (missing ? (int)(p >> 31) : 0) <= spare) open |= 1u << out;
    }
    return open;
}

// Best replacement of one cut: the body of EvaluateNode's cut loop
// (src/algorithms/rewrite.cu:386-445).  Returns the first root (in root
// order) with the highest gain and, among equal gains, the lowest level:
// out < 0 when no root qualifies.
struct CutBest {
    int gain, level, out;
};

// saved is CalcMFFC's count for this cut, del its nDel MFFC nodes (the table
// entries whose count reached zero), least the smallest gain that counts and
// roots the ones to consider (the others cannot qualify).
//
// A library node can be matched only when both its fanins are, to nodes
// other than q and its MFFC.  So the walk starts from the input pairs whose
// AND the filters leave possible, and goes on through the readers of each
// matched node, in index order (fanins precede their node): the nodes that it
// does not reach are those that the reference's loop over the whole forest
// (rewrite.cu:400-428) leaves unmatched.
//
// No level is kept: a matched node's fanins are the nodes its library fanins
// are matched to, so every library node, matched or not, is one level above
// the higher of its fanins, and a root's level follows from the inputs'
// levels and its longest paths to them.
CULS_HD CutBest eval_cut(const EvalIn &E, int q, const CutView &v, uint32_t roots, int least, int saved, int nDel,
                         const int *del) {
    CutBest best{-1, 0, -1};
    const int cls = v.cls;
    int match[kMaxLibNodes];
    uint64_t cones = 0;
    for (uint32_t m = roots; m; m &= m - 1) cones |= E.lib->rootCone[cls][ctz64(m)];
    uint64_t todo = E.lib->pairRest[cls];
    for (uint32_t p = v.possible; p; p &= p - 1) todo |= 1ull << E.lib->pairNode[cls][ctz64(p)];
    todo &= cones;
    uint64_t have = 15, self = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) match[j] = v.in[j];
    while (todo) {
        const int n = ctz64(todo);
        todo &= todo - 1;
        const uint32_t w = E.lib->node[cls][n - 4];
        const int in0 = ln_f0(w), in1 = ln_f1(w);
        if (!((have >> in0) & (have >> in1) & 1ull)) continue;
        const int cc0 = (in0 < 4 ? ((v.isC >> in0) & 1) : 0) ^ ln_c0(w);
        const int cc1 = (in1 < 4 ? ((v.isC >> in1) & 1) : 0) ^ ln_c1(w);
        const int r = region_and_lookup(E.tab, match[in0], match[in1], cc0, cc1, E.status);
        if (r == -1 || mffc_member(r, nDel, del)) continue;
        if (r == q) {
            self |= 1ull << n;
        } else {
            match[n] = r;
            have |= 1ull << n;
            todo |= E.lib->uses[cls][n] & cones;
        }
    }
    // Nodes a root adds (Eval, rewrite.cu:369-374): the unmatched ones of its
    // cone.  A node is matched only when both its fanins are (inputs always
    // are), so a matched node's whole cone is matched and every unmatched node
    // of the cone is reached through unmatched nodes.
    const uint64_t missing = ~(have | self);
    for (uint32_t m = roots; m; m &= m - 1) {
        const int out = ctz64(m);
        const int gain = saved - popc64(E.lib->rootCone[cls][out] & missing);
        if (gain < best.gain || gain < least) continue;
        if ((self >> E.lib->roots[cls][out]) & 1ull) continue;
        const uint32_t depth = E.lib->rootDepth[cls][out];
        int level = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int d = (int)((depth >> (8 * j)) & 255u), x = E.level[v.in[j]] + d - 1;
            level = d && x > level ? x : level;
        }
        if (best.out >= 0 && gain == best.gain && level >= best.level) continue;
        best = CutBest{gain, level, out};
    }
    return best;
}

// EvaluateNode's choice across cuts (src/algorithms/rewrite.cu:378-447):
// cuts in slot order, a later cut wins only with a higher gain or an equal
// gain at a lower level.  Folds cut i's best into (bestCut, bestOut, gain,
// level).
CULS_HD void fold_cut_best(const CutBest &c, int i, int &bestCut, int &bestOut, int &gain, int &level) {
    if (c.out < 0) return;
    if (bestCut >= 0 && (c.gain < gain || (c.gain == gain && c.level >= level))) return;
    bestCut = i;
    bestOut = c.out;
    gain = c.gain;
    level = c.level;
}

}  // namespace culs
