"""The rewrite's scratch is sized by the graph's objects before the number of
replacement records is known.  A design with millions of copies of one block
over the same inputs has nearly as many records as nodes, most of which merge:
it must still fit, and give the oracle's graph."""
import numpy as np
import pytest

import culs_b200 as C
from oracle.oracle import Oracle
from util import same_graph, to_oracle

pytestmark = pytest.mark.gpu

# ten ANDs over six inputs: six of them have a replacement, of ten nodes in all
BLOCK = ([5, 5, 10, 10, 13, 16, 15, 16, 26, 21], [13, 6, 12, 14, 14, 19, 24, 22, 29, 31])


def blocks(count):
    n0, n = 7, len(BLOCK[0])
    shift = 2 * n * np.arange(count, dtype=np.int32)[:, None]
    fanins = [np.where(x >> 1 >= n0, x + shift, x + 0 * shift).reshape(-1) for x in np.array(BLOCK, np.int32)]
    pad = np.full(n0, -1, np.int32)
    return C.Aig(6, *[np.concatenate([pad, x]).astype(np.int32) for x in fanins],
                 (2 * (n0 + n - 1 + n * np.arange(count))).astype(np.int32))


@pytest.mark.parametrize("count", [3000, 550000])
def test_many_duplicate_replacements_fit_and_match_oracle(count):
    g = blocks(count)
    o = Oracle()
    o.set_graph(to_oracle(g))
    o.rw(zeros=True)
    ctx = C.Context()
    try:
        d = ctx.upload(g)
        ctx.rw(d, zeros=True)
        assert same_graph(d.download(), o.graph())
        assert ctx.rw_stats()["replaced"] == o.dump_stats()["replaced"] >= count
    finally:
        ctx.close()
