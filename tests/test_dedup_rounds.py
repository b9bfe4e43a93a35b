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
