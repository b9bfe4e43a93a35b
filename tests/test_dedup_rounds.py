"""The strash's hashing in rounds (CULS_DEDUP_MODE=rounds) keys, after its
first round, only the nodes whose fanins' mapping changed.  Copies of a graph
merge level by level, so the rounds cascade as deep as the copies are; a table
with little room for the later rounds' keys makes them start again from all
nodes.  Every way must give the oracle's graph, also in id order (`st -c`)."""
import numpy as np
import pytest

import culs_b200 as C
from oracle.oracle import Oracle
from util import same_graph, to_oracle

pytestmark = pytest.mark.gpu


def copies(g, k, shuffle_seed=None):
    """k structural copies of g over the same PIs, all outputs kept; the
    copies' nodes interleaved at random when a seed is given."""
    n0 = 1 + g.nPIs
    parts = []
    for c in range(k):
        shift = c * g.nAnds
        f = [np.where((x >> 1) >= n0, x + 2 * shift, x) for x in (g.fanin0[n0:], g.fanin1[n0:])]
        parts.append((f[0], f[1], np.where((g.outs >> 1) >= n0, g.outs + 2 * shift, g.outs)))
    f0, f1, outs = (np.concatenate([p[i] for p in parts]) for i in range(3))
    if shuffle_seed is not None:
        rng = np.random.default_rng(shuffle_seed)
        key = np.concatenate([np.sort(rng.random(g.nAnds)) for _ in range(k)])
        order = np.argsort(key, kind="stable")
        new = np.empty(len(order), np.int64)
        new[order] = np.arange(len(order))
        ren = lambda x: np.where((x >> 1) >= n0, 2 * (n0 + new[np.maximum((x >> 1) - n0, 0)]) + (x & 1), x)  # noqa: E731
        f0, f1, outs = ren(f0)[order], ren(f1)[order], ren(outs)
        f0, f1 = np.minimum(f0, f1), np.maximum(f0, f1)
    pad = np.full(n0, -1)
    return C.Aig(g.nPIs, *[np.concatenate([pad, x]).astype(np.int32) for x in (f0, f1)], outs.astype(np.int32))


def graphs():
    deep = C.gen_layered(5, 16, 8, 1500, 45, 3, 0.1, True)
    return [copies(C.gen_multiplier(6), 2), copies(C.gen_multiplier(10), 3, 1), copies(deep, 2, 2), copies(deep, 5, 3)]


@pytest.mark.parametrize("room", [None, 1.0, 1.2])
@pytest.mark.parametrize("cpu", [False, True])
def test_cascading_merges_match_oracle(cpu, room, monkeypatch):
    ctx = C.Context()
    try:
        for i, g in enumerate(graphs()):
            o = Oracle()
            o.set_graph(to_oracle(g))
            o.st(cpu=cpu)
            ref = o.graph()
            assert ref.nAnds < g.nAnds
            if room is None:
                monkeypatch.delenv("CULS_STRASH_TABLE_CAP", raising=False)
            else:  # rounded up to a power of two: load 1/2 to 1
                monkeypatch.setenv("CULS_STRASH_TABLE_CAP", str(int(room * g.nAnds)))
            for mode in ["rounds", "levels"]:
                monkeypatch.setenv("CULS_DEDUP_MODE", mode)
                d = ctx.upload(g)
                ctx.st(d, cpu=cpu)
                got = d.download()
                assert same_graph(got, ref) and got.nLevels == ref.nLevels, (i, mode)
    finally:
        ctx.close()


def test_batch_of_copies_matches_oracle(monkeypatch):
    gs = graphs() * 3
    ctx = C.Context()
    try:
        d = ctx.upload_batch(gs)
        ctx.rw_st(d)
        for g, got in zip(gs, d.download_all()):
            o = Oracle()
            o.set_graph(to_oracle(g))
            o.rw()
            o.st()
            assert same_graph(got, o.graph())
    finally:
        ctx.close()


def readers_of_a_duplicate(n):
    """At most n ANDs: a node and its duplicate, a ladder of nodes none alike,
    and one reader of the duplicate over each of those, which all get another
    key when the duplicate has merged."""
    n_pis, m = 40, (n - 2) // 2
    first = 1 + n_pis  # the node, its duplicate, the ladder, the readers
    v = np.arange(m)
    f0 = 2 * (1 + v % n_pis) + (v // n_pis & 1)
    f1 = np.where(v < 3, 2 * (1 + (v + 1) % n_pis), 2 * (first + 2 + v - 3) + 1)
    r0, r1 = np.full(m, 2 * (first + 1)), 2 * (first + 2 + v)
    pad, pair = np.full(first, -1), np.array([2, 2])
    f0, f1 = np.concatenate([pad, pair, f0, r0]), np.concatenate([pad, pair + 2 * 7, f1, r1])
    return C.Aig(n_pis, np.minimum(f0, f1).astype(np.int32), np.maximum(f0, f1).astype(np.int32),
                 np.append(2 * (first + 2 + m + v), 2 * first).astype(np.int32))


@pytest.mark.parametrize("cap,n", [(4096, 4096), (4096, 4094), (4096, 3900), (64, 64), (64, 50), (4096, 2048)])
def test_a_table_with_room_for_every_node_is_enough(cap, n, monkeypatch):
    """A table that the level dataflow gets along with does for the rounds
    too, although their later rounds make further keys."""
    g = readers_of_a_duplicate(n)
    assert n - 1 <= g.nAnds <= n
    o = Oracle()
    o.set_graph(to_oracle(g))
    o.st()
    assert o.graph().nAnds == g.nAnds - 1
    monkeypatch.setenv("CULS_STRASH_TABLE_CAP", str(cap))
    ctx = C.Context()
    try:
        for mode in ["levels", "rounds"]:
            monkeypatch.setenv("CULS_DEDUP_MODE", mode)
            d = ctx.upload(g)
            ctx.st(d)
            assert same_graph(d.download(), o.graph()), mode
    finally:
        ctx.close()
