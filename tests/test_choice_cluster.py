"""The choice loop (CULS src/algorithms/rewrite.cu:830-921) gives each graph
a block, or, where at most 18 graphs have 1,024 candidates each on average, a
cluster of eight blocks, and replays their candidates in windows;
CULS_CHOICE_GLOBAL replays every candidate alone on the graph instead.  Each
way must give the oracle's graph, with the same choice statistics."""
import pytest

import culs_b200 as C
from oracle.oracle import Oracle
from test_choice_windows import STATS, carry_chains
from util import same_graph, to_oracle

pytestmark = pytest.mark.gpu


def graphs():
    return [
        C.gen_multiplier(4),  # a block
        C.gen_multiplier(16),
        C.gen_multiplier(64),  # a cluster
        C.gen_layered(11, 64, 32, 60000, 120, 4, 0.0, True),
        C.gen_layered(13, 128, 64, 130000, 160, 4, 0.0, True),
    ]


def oracle(g, zeros):
    o = Oracle()
    o.set_graph(to_oracle(g))
    o.rw(zeros=zeros)
    o.st()
    return o.graph(), o.dump_stats()


@pytest.mark.parametrize("zeros", [False, True])
def test_cluster_choice_matches_oracle_and_global_walk(zeros, monkeypatch):
    ctx = C.Context()
    try:
        for i, g in enumerate(graphs()):
            got = {}
            for mode in ["cluster", "global"]:
                if mode == "global":
                    monkeypatch.setenv("CULS_CHOICE_GLOBAL", "1")
                else:
                    monkeypatch.delenv("CULS_CHOICE_GLOBAL", raising=False)
                d = ctx.upload(g)
                ctx.rw(d, zeros=zeros)
                st = ctx.rw_stats()
                ctx.st(d)
                got[mode] = (d.download(), st)
                d.free()
            ref, rs = oracle(g, zeros)
            assert same_graph(got["cluster"][0], ref), i
            assert same_graph(got["global"][0], ref), i
            for k in ["replaced", "replaced_pos", "replaced_zero", "reverted", "compromised"]:
                assert got["cluster"][1][k] == got["global"][1][k] == rs[k], (i, k)
    finally:
        ctx.close()


def replacements(st):
    return st["candidates"] - st["new_idx"]


@pytest.mark.parametrize("bits,cluster", [(342, False), (343, True)])
def test_both_sides_of_the_line_match_oracle(bits, cluster):
    g = carry_chains(1, bits, False)
    ref, rs = oracle(g, True)
    ctx = C.Context()
    try:
        d = ctx.upload(g)
        ctx.rw(d, zeros=True)
        st = ctx.rw_stats()
        assert abs(replacements(st) - 1024) <= 3 and (replacements(st) >= 1024) == cluster
        ctx.st(d)
        assert same_graph(d.download(), ref) and {k: st[k] for k in STATS} == {k: rs[k] for k in STATS}
    finally:
        ctx.close()


@pytest.mark.parametrize("first", [0, 2, 3])
def test_several_graphs_on_clusters_match_oracle(first):
    """Graphs of very different numbers of candidates, each on its cluster."""
    gs = [C.gen_multiplier(8), C.gen_multiplier(48), C.gen_layered(11, 64, 32, 60000, 120, 4, 0.0, True),
          carry_chains(2, 400, False), carry_chains(30, 40, True), C.gen_multiplier(2)][first:]
    ctx = C.Context()
    try:
        for zeros in [False, True]:
            d = ctx.upload_batch(gs)
            ctx.rw(d, zeros=zeros)
            st = ctx.rw_stats()
            assert not zeros or replacements(st) >= 1024 * len(gs)
            ctx.st(d)
            want = dict.fromkeys(STATS, 0)
            for g, got in zip(gs, d.download_all()):
                ref, rs = oracle(g, zeros)
                assert same_graph(got, ref)
                for k in STATS:
                    want[k] += rs[k]
            assert {k: st[k] for k in STATS} == want
    finally:
        ctx.close()
