"""The balance (CULS src/algorithms/balance.cu:912-1382) works on a graph
with a block, a thread-block cluster or the whole grid, by its width, and on
the graphs of a batch together as far as scratch allows.  Graphs whose levels
are about as wide as each team, covers longer than a thread keeps (32 leaves)
and than the reference's limits, constant covers, and a budget that takes the
graphs one at a time must all give the oracle's graph."""
import numpy as np
import pytest

import culs_b200 as C
from oracle.oracle import Oracle
from util import same_graph, to_oracle

pytestmark = pytest.mark.gpu


def oracle_b(g):
    o = Oracle()
    o.set_graph(to_oracle(g))
    o.b()
    return o.graph()


def check(ctx, g):
    d = ctx.upload(g)
    ctx.b(d)
    got, ref = d.download(), oracle_b(g)
    assert same_graph(got, ref) and got.nLevels == ref.nLevels


def products(seed, n_pis, sizes, contradict=False):
    """Single-fanout AND chains of the given sizes over random PI literals,
    their outputs paired up; with `contradict`, every third chain holds a
    literal and its complement."""
    rng = np.random.default_rng(seed)
    f0, f1 = [-1] * (1 + n_pis), [-1] * (1 + n_pis)

    def new(a, b):
        f0.append(min(a, b))
        f1.append(max(a, b))
        return 2 * (len(f0) - 1)

    tops = []
    for k, size in enumerate(sizes):
        lits = [int(2 * p + rng.integers(0, 2)) for p in rng.choice(np.arange(1, 1 + n_pis), size, replace=False)]
        if contradict and k % 3 == 0:
            lits[-1] = lits[0] ^ 1
        x = lits[0]
        for y in lits[1:]:
            x = new(x, y)
        tops.append(x)
    outs = [new(a ^ 1, b ^ 1) for a, b in zip(tops, tops[1:])] + tops[:1]
    return C.Aig(n_pis, np.array(f0, np.int32), np.array(f1, np.int32), np.array(outs, np.int32))


@pytest.fixture(scope="module")
def ctx():
    c = C.Context()
    yield c
    c.close()


@pytest.mark.parametrize("ands,layers", [(4000, 10), (6000, 10), (11000, 10), (22000, 10), (45000, 10), (90000, 20),
                                         (120000, 10)])
def test_every_team_matches_oracle(ctx, ands, layers):
    check(ctx, C.gen_layered(3, 600, 400, ands, layers, 3, 0.1, True))


@pytest.mark.parametrize("contradict", [False, True])
@pytest.mark.parametrize("longest", [31, 33, 120, 140, 1030])
def test_long_covers_match_oracle(ctx, longest, contradict):
    rng = np.random.default_rng(longest)
    sizes = [int(s) for s in rng.integers(2, longest, 40)] + [longest, longest - 1, 2, 32]
    check(ctx, products(longest, 1100, sizes, contradict))


def test_batch_and_tight_budget_match_oracle(ctx):
    gs = [C.gen_multiplier(20), C.gen_layered(3, 600, 400, 22000, 10, 3, 0.1, True), products(1, 200, [5, 60, 3, 150]),
          C.gen_multiplier(3), *C.gen_batch(4, 10, 20, 200, 5000, 16, 64, threads=8)]
    refs = [oracle_b(g) for g in gs]
    largest = max(g.nObjs for g in gs)
    tight = C.Context(hbm_budget=largest * 900 + (200 << 20))
    try:
        for c in [ctx, tight]:
            d = c.upload_batch(gs)
            c.b(d)
            for i, ref in enumerate(refs):
                got = d.download(i)
                assert same_graph(got, ref) and got.nLevels == ref.nLevels, i
    finally:
        tight.close()


def caterpillar(n_pis, length, seed, repeat):
    """Chains x = x & (p & q) whose pair nodes come after the chain's node, so
    that a cover's DFS has every pair waiting on its stack; with `repeat`, the
    pairs' literals recur (a leaf met again, or its complement)."""
    rng = np.random.default_rng(seed)
    f0, f1, outs = [-1] * (1 + n_pis), [-1] * (1 + n_pis), []

    def new(a, b):
        f0.append(min(a, b))
        f1.append(max(a, b))
        return 2 * (len(f0) - 1)

    for k in range(60):
        pool = iter(rng.permutation(np.arange(1, 1 + n_pis)))
        x = 2 * int(next(pool))
        for i in range(length if k % 4 else 40):
            if repeat and i % 7 == 3:
                p = int(rng.integers(1, 1 + n_pis))
                q = 1 + (p + int(rng.integers(0, n_pis - 1))) % n_pis
                x = new(x, new(2 * p, 2 * q))
            else:
                x = new(x, new(*[int(2 * next(pool) + (0 if repeat else rng.integers(0, 2))) for _ in range(2)]))
        outs.append(x)
    return C.Aig(n_pis, np.array(f0, np.int32), np.array(f1, np.int32), np.array(outs, np.int32))


@pytest.mark.parametrize("length", [17, 60, 125, 127, 128, 200, 510])
def test_deep_stacks_and_repeated_leaves_match_oracle(ctx, length):
    check(ctx, caterpillar(1100, length, length, False))
    check(ctx, caterpillar(1100, length, length, True))


@pytest.mark.parametrize("count,size", [(700, 34), (3000, 100), (300, 400)])
def test_many_long_covers_at_once_match_oracle(ctx, count, size):
    check(ctx, products(7, 600, [size] * count))


def no_ands(n_pis, n_pos):
    pad = np.full(1 + n_pis, -1, np.int32)
    return C.Aig(n_pis, pad, pad.copy(), (np.arange(n_pos) % (2 + 2 * n_pis)).astype(np.int32))


def test_graphs_without_and_nodes_match_oracle(ctx):
    """Alone, a batch of them, and among others, together and one at a time."""
    check(ctx, no_ands(3, 8))
    check(ctx, no_ands(1, 0))
    gs = [no_ands(5, 4), C.gen_multiplier(6), no_ands(2, 1), C.gen_layered(3, 600, 400, 22000, 10, 3, 0.1, True),
          no_ands(300, 700)]
    tight = C.Context(hbm_budget=max(g.nObjs for g in gs) * 900 + (200 << 20))
    try:
        for c in [ctx, tight]:
            for batch in [gs, gs[:1] + gs[2:3] + gs[4:], gs[::-1]]:
                d = c.upload_batch(batch)
                c.b(d)
                for g, got in zip(batch, d.download_all()):
                    ref = oracle_b(g)
                    assert same_graph(got, ref) and got.nLevels == ref.nLevels
    finally:
        tight.close()
