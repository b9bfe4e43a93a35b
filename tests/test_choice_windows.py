"""The choice loop (CULS src/algorithms/rewrite.cu:830-921) takes a graph's
candidates a window at a time, one per thread, and commits the part of the
window that no earlier candidate disturbs.  The cases here are where that can
go wrong: candidates that touch more nodes than a thread's overlay holds, or
nest deeper than its stack (both are replayed alone), windows that the
candidates just fill, and the numbers of graphs at which a block's width
changes.  All must give the oracle's graph and choice statistics exactly."""
import numpy as np
import pytest

import culs_b200 as C
from oracle.oracle import Oracle
from util import same_graph, to_oracle

pytestmark = pytest.mark.gpu
STATS = ["replaced", "replaced_pos", "replaced_zero", "reverted", "compromised", "new_idx", "expected"]


def oracle(g, zeros):
    o = Oracle()
    o.set_graph(to_oracle(g))
    o.rw(zeros=zeros)
    st = o.dump_stats()
    o.st()
    return o.graph(), st


def redundant_cones(n, cones, balanced):
    """Per cone, ((a & b) | (a & !b)) & (c | d) = a & (c | d) over a b that is a
    cone of n inputs used nowhere else: the replacement deletes all of b."""
    n_pis = 3 + n * cones
    f0, f1 = [-1] * (1 + n_pis), [-1] * (1 + n_pis)
    a, c, d = 2, 4, 6
    pi = iter(range(4, 1 + n_pis))

    def new(x, y):
        f0.append(min(x, y))
        f1.append(max(x, y))
        return 2 * (len(f0) - 1)

    outs = []
    for _ in range(cones):
        lits = [2 * next(pi) for _ in range(n)]
        if balanced:
            while len(lits) > 1:
                lits = [new(lits[i], lits[i + 1]) for i in range(0, len(lits) - 1, 2)] + lits[len(lits) & ~1:]
            b = lits[0]
        else:
            b = lits[0]
            for x in lits[1:]:
                b = new(b, x)
        x = new(new(a, b) ^ 1, new(a, b ^ 1) ^ 1) ^ 1
        outs.append(new(x, new(c ^ 1, d ^ 1) ^ 1))
    return C.Aig(n_pis, np.array(f0, np.int32), np.array(f1, np.int32), np.array(outs, np.int32))


@pytest.fixture(scope="module")
def ctx():
    c = C.Context()
    yield c
    c.close()


@pytest.mark.parametrize("balanced", [False, True])
@pytest.mark.parametrize("n", [3, 7, 15, 16, 17, 30, 33, 70, 200])
def test_large_deletions_match_oracle(ctx, n, balanced):
    g = redundant_cones(n, 5, balanced)
    for zeros in [False, True]:
        ref, rs = oracle(g, zeros)
        assert rs["replaced"] >= 1 and rs["expected"] >= n
        d = ctx.upload(g)
        ctx.rw(d, zeros=zeros)
        st = ctx.rw_stats()
        ctx.st(d)
        assert same_graph(d.download(), ref), zeros
        assert {k: st[k] for k in STATS} == {k: rs[k] for k in STATS}, zeros


@pytest.mark.parametrize("count", [1, 2, 147, 149, 443, 445])
def test_every_block_width_matches_oracle(ctx, count):
    gs = C.gen_batch(9, 0, count, 100, 1500, 8, 64, threads=8)
    d = ctx.upload_batch(gs)
    ctx.rw(d, zeros=True)
    total = ctx.rw_stats()
    ctx.st(d)
    out = d.download_all()
    want = dict.fromkeys(STATS, 0)
    for g, r in zip(gs, out):
        ref, rs = oracle(g, True)
        assert same_graph(r, ref)
        for k in STATS:
            want[k] += rs[k]
    assert {k: total[k] for k in STATS} == want


def carry_chains(chains, bits, xors):
    """Ripple carry adders of majority gates, or (xors) chains of two-input
    exclusive ors in two forms: every stage's replacement changes what the next
    stage's reads, so that windows commit hardly more than one candidate."""
    n_pis = 2 * bits * chains
    f0, f1, outs = [-1] * (1 + n_pis), [-1] * (1 + n_pis), []

    def land(a, b):
        f0.append(min(a, b))
        f1.append(max(a, b))
        return 2 * (len(f0) - 1)

    def lor(a, b):
        return land(a ^ 1, b ^ 1) ^ 1

    def xor(a, b, form=0):
        return land(lor(a, b), land(a, b) ^ 1) if form else lor(land(a, b ^ 1), land(a ^ 1, b))

    for k in range(chains):
        first = 1 + 2 * bits * k
        c = land(2 * first, 2 * first + 2)
        for i in range(1, bits):
            x, y = 2 * (first + 2 * i), 2 * (first + 2 * i + 1)
            if xors:
                c = xor(xor(c, x, i & 1), y, ~i & 1)
                continue
            outs.append(xor(xor(x, y), c))
            c = lor(lor(land(x, y), land(x, c)), land(y, c))
        outs.append(c)
    return C.Aig(n_pis, np.array(f0, np.int32), np.array(f1, np.int32), np.array(outs, np.int32))


@pytest.mark.parametrize("xors", [False, True])
@pytest.mark.parametrize("graphs,chains,bits", [(1, 1, 5), (1, 1, 60), (1, 1, 700), (1, 3, 300), (3, 1, 600), (40, 1, 33),
                                                (160, 2, 12), (460, 1, 20)])
def test_dependent_candidates_match_oracle(ctx, graphs, chains, bits, xors):
    g = carry_chains(chains, bits, xors)
    for zeros in [False, True]:
        ref, rs = oracle(g, zeros)
        assert not zeros or rs["replaced"] >= 1
        d = ctx.upload_batch([g] * graphs) if graphs > 1 else ctx.upload(g)
        ctx.rw(d, zeros=zeros)
        st = ctx.rw_stats()
        ctx.st(d)
        assert all(same_graph(r, ref) for r in (d.download_all() if graphs > 1 else [d.download()])), zeros
        assert {k: st[k] for k in STATS} == {k: graphs * rs[k] for k in STATS}, zeros


def hub_cones(n, drop, extra):
    """n cones over one AND node h and inputs of their own, ((h & b) | (h & !b))
    & (c | d) = h & (c | d), each replacement taking one of h's two references
    away, or with `drop` ((h & b) | (!h & b)) & (c | d) = b & (c | d), both of
    them, so that the last replacement deletes h; `extra` more references from
    outputs."""
    n_pis = 2 + 3 * n
    f0, f1, outs = [-1] * (1 + n_pis), [-1] * (1 + n_pis), []

    def new(a, b):
        f0.append(min(a, b))
        f1.append(max(a, b))
        return 2 * (len(f0) - 1)

    h = new(2, 4)
    for i in range(n):
        b, c, d = [2 * (3 + 3 * i + k) for k in range(3)]
        x = new(new(h, b) ^ 1, new(h ^ drop, b ^ 1 ^ drop) ^ 1) ^ 1
        outs.append(new(x, new(c ^ 1, d ^ 1) ^ 1))
    return C.Aig(n_pis, np.array(f0, np.int32), np.array(f1, np.int32), np.array(outs + [h] * extra, np.int32))


@pytest.mark.parametrize("drop", [0, 1])
@pytest.mark.parametrize("n,extra", [(1, 0), (126, 2), (127, 0), (127, 1), (127, 2), (127, 3), (128, 2), (200, 1), (510, 1),
                                     (511, 0), (511, 1), (512, 0), (600, 0), (1100, 0), (1100, 3000), (3000, 0), (3000, 1)])
def test_a_node_with_many_references_matches_oracle(ctx, n, extra, drop):
    """Reference counts around 255, where the MFFC count of a node saturates,
    and around 1,022, where the lowest count that mattered to a candidate does;
    windows that take more references away than that."""
    g = hub_cones(n, drop, extra)
    for zeros in [False, True]:
        ref, rs = oracle(g, zeros)
        assert rs["replaced"] >= n
        d = ctx.upload(g)
        ctx.rw(d, zeros=zeros)
        st = ctx.rw_stats()
        ctx.st(d)
        assert same_graph(d.download(), ref), zeros
        assert {k: st[k] for k in STATS} == {k: rs[k] for k in STATS}, zeros
