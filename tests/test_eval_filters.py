"""Evaluation (CULS src/algorithms/rewrite.cu:378-471) reaches a library node
only through matched fanins, starting from the input pairs that the nodes'
64-bit filters leave possible, and drops the roots whose cones lack too many
pairs.  The graphs here have few inputs (filters with every bit set), many
(hardly any), constants as cut leaves, duplicate nodes and both kinds of MFFC;
the selected cut, root and gain of every node must equal the oracle's, with
and without zero-gain replacements."""
import numpy as np
import pytest

import culs_b200 as C
from oracle.oracle import Oracle
from test_enum_forms import random_aig
from util import to_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zeros", [False, True])
@pytest.mark.parametrize("n_pis,n_ands,reach", [(3, 100, 100), (4, 1500, 30), (5, 3000, 3000), (12, 3000, 40),
                                                (200, 4000, 400), (1000, 1500, 100)])
def test_selected_cuts_match_oracle(n_pis, n_ands, reach, zeros):
    ctx = C.Context()
    try:
        for seed in range(10, 12):
            g = random_aig(seed, n_pis, n_ands, reach)
            o = Oracle()
            o.set_graph(to_oracle(g))
            o.rw(zeros)
            ctx.rw(ctx.upload(g), zeros, dump=True)
            np.testing.assert_array_equal(ctx.dump()["selected"].reshape(-1, 10), o.dump_selected())
    finally:
        ctx.close()
