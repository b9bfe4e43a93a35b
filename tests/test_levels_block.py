"""Levels of a single graph of up to 57,000 nodes come from one block's shared
memory, larger ones from the dataflow over global memory; the rewrite's
deduplication passes nodes of its order that a reused later node leaves
unresolved.  Sizes around a row of threads and around the bound, the deepest
and the flattest graphs, dangling nodes and consecutive rewrites (whose kept
graphs are out of order) must all give the oracle's graph and levels."""
import numpy as np
import pytest

import culs_b200 as C
from oracle.oracle import Oracle
from util import same_graph, to_oracle

pytestmark = pytest.mark.gpu


def chain(n_ands, dangling):
    """A chain of ANDs over alternating PIs; with `dangling`, every other PO
    is on an early node, so the rest of the chain hangs."""
    n_pis = 3
    v = np.arange(n_ands, dtype=np.int32)
    f0 = np.concatenate([np.full(4, -1), np.where(v == 0, 2, 2 * (1 + v % 3))]).astype(np.int32)
    f1 = np.concatenate([np.full(4, -1), np.where(v == 0, 4, 2 * (3 + v) + 1)]).astype(np.int32)
    top = 4 + (n_ands // 2 if dangling else n_ands - 1)
    return C.Aig(n_pis, f0, f1, np.array([2 * top, 2 * 4 + 1], np.int32))


def flat(n_ands, k=400):
    """n_ands ANDs of two of the k PIs each."""
    i, j = np.triu_indices(k, 1)
    f0 = np.concatenate([np.full(1 + k, -1), 2 * (1 + i[:n_ands])]).astype(np.int32)
    f1 = np.concatenate([np.full(1 + k, -1), 2 * (1 + j[:n_ands])]).astype(np.int32)
    return C.Aig(k, f0, f1, 2 * np.arange(1 + k, 1 + k + n_ands, dtype=np.int32))


def check(ctx, g, dedup=2, twice=False):
    o = Oracle()
    o.set_graph(to_oracle(g))
    d = ctx.upload(g)
    for _ in range(2 if twice else 1):
        o.rw(dedup=dedup)
        ctx.rw(d, gpu_dedup=dedup == 2)
    mid, want = d.download(), o.graph()
    assert same_graph(mid, want) and mid.nLevels == want.nLevels
    o.st()
    ctx.st(d)
    got, want = d.download(), o.graph()
    assert same_graph(got, want) and got.nLevels == want.nLevels


@pytest.fixture(scope="module")
def ctx():
    c = C.Context()
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1019, 1020, 1021, 2045, 5000])
def test_rows_of_threads(ctx, n):
    for g in [chain(n, False), chain(n, True), flat(n)]:
        check(ctx, g)


@pytest.mark.parametrize("objs", [56999, 57000, 57001])
def test_around_the_bound(ctx, objs):
    g = flat(objs - 401)
    assert g.nObjs == objs
    check(ctx, g)


@pytest.mark.parametrize("dedup,twice", [(2, True), (1, False), (1, True)])
def test_unresolved_nodes_of_the_order(ctx, dedup, twice):
    for g in [C.gen_multiplier(24), C.gen_multiplier(64), C.gen_layered(7, 64, 32, 30000, 60, 4, 0.0, True)]:
        check(ctx, g, dedup, twice)
