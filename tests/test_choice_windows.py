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
