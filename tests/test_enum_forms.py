"""Cut enumeration (CULS src/algorithms/rewrite.cu:268-294) runs a level's
nodes one per thread or one per warp, by the level's width; the warp form
replays the slot policy on precomputed containment bits.  The graphs here have
nodes with every number of admissible fanin-cut pairs up to 64 (few inputs, so
that most pairs fit four leaves), cuts that shrink under minimisation down to
none, and duplicate and constant nodes; every cut slot must equal the
oracle's, whichever form each level takes."""
import numpy as np
import pytest

import culs_b200 as C
from oracle.oracle import Oracle
from util import to_oracle

pytestmark = pytest.mark.gpu


def random_aig(seed, n_pis, n_ands, reach):
    """Fanins among the PIs and the last `reach` nodes, any phases; some
    constant fanins, equal fanins and duplicate nodes."""
    rng = np.random.default_rng(seed)
    n = 1 + n_pis + n_ands
    f0, f1 = np.full(n, -1, np.int32), np.full(n, -1, np.int32)
    for v in range(1 + n_pis, n):
        r = rng.random()
        if r < 0.03 and v > 2 + n_pis:
            u = int(rng.integers(1 + n_pis, v))
            f0[v], f1[v] = f0[u], f1[u]
            continue
        lo = max(1, v - reach)
        a, b = [int(2 * (rng.integers(lo, v) if rng.random() < 0.7 else rng.integers(1, 1 + n_pis)) + rng.integers(0, 2))
                for _ in range(2)]
        if r < 0.05:
            a = int(rng.integers(0, 2))
        elif r < 0.07:
            b = a ^ int(rng.integers(0, 2))
        f0[v], f1[v] = min(a, b), max(a, b)
    outs = 2 * np.arange(max(1, n - 40), n, dtype=np.int32)
    return C.Aig(n_pis, f0, f1, outs)


@pytest.mark.parametrize("wide_min", [1, 4, 1 << 30])
@pytest.mark.parametrize("n_pis,n_ands,reach", [(2, 60, 60), (3, 200, 12), (4, 800, 30), (4, 1500, 1500), (5, 1500, 20),
                                                (6, 2000, 200), (9, 3000, 60), (40, 3000, 300)])
def test_every_cut_slot_matches_oracle(n_pis, n_ands, reach, wide_min):
    ctx = C.Context()
    try:
        ctx.set_param("enum_wide_min", wide_min)
        for seed in range(2):
            g = random_aig(seed, n_pis, n_ands, reach)
            o = Oracle()
            o.set_graph(to_oracle(g))
            o.rw()
            d = ctx.upload(g)
            ctx.rw(d, dump=True)
            D = ctx.dump()
            np.testing.assert_array_equal(D["cuts"].reshape(-1, 8, 9), o.dump_cuts())
            np.testing.assert_array_equal(D["selected"].reshape(-1, 10), o.dump_selected())
    finally:
        ctx.close()


@pytest.mark.parametrize("name", ["mult48", "deep"])
def test_records_are_read_after_their_node_is_ready(name):
    """Deep graphs, where a node's fanins become ready on another SM while its
    warp waits for them: two lanes wait, the others read the fanins' records.
    Repeated, as a read that came too early would not come so every time."""
    g = C.gen_multiplier(48) if name == "mult48" else C.gen_layered(3, 40, 20, 20000, 400, 2, 0.0, True)
    o = Oracle()
    o.set_graph(to_oracle(g))
    o.rw()
    cuts, selected = o.dump_cuts(), o.dump_selected()
    ctx = C.Context()
    try:
        for _ in range(6):
            ctx.rw(ctx.upload(g), dump=True)
            D = ctx.dump()
            np.testing.assert_array_equal(D["cuts"].reshape(-1, 8, 9), cuts)
            np.testing.assert_array_equal(D["selected"].reshape(-1, 10), selected)
    finally:
        ctx.close()
