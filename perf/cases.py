"""The work that programs using this framework have it do, as measurable cases.

A case is a family of AIGs, how they reach the framework and a list of
commands, named as the reference's command line names them (`rw`, `rw -z`,
`st`, `st -c`, `b`; `rw -c` is the rewrite with CPU deduplication that the
ABC-patch `grw` runs by default).

How the graphs reach the framework:
  resident  device handles kept by the program; the commands run on a clone,
            so that the input stays, and the result is downloaded
  host      AIGMan arrays in host memory, uploaded, processed and downloaded
  aiger     binary AIGER bytes in host memory, decoded and encoded on the GPU
  served    jobs submitted to the served mode's workers and fetched

Every output is an integer array that the commands determine completely.
"""
import ctypes
import functools
import math

import numpy as np

import culs_b200 as C


def listed():
    return [
        # one small block: what latency, launches and host round trips cost
        dict(name="mult8_rw_st", family="mult", n=8, path="resident", commands="rw; st"),
        # an ordinary control-logic sized block
        dict(name="layered5k_rw_st", family="layered", pis=64, pos=32, ands=5000, layers=40, window=4, far=0.0,
             from_pis=True, path="resident", commands="rw; st"),
        # a deep arithmetic block, the repository's single-graph benchmark
        dict(name="mult64_rw_st", family="mult", n=64, path="resident", commands="rw; st"),
        # an optimisation script: resyn2 without its refactoring steps
        dict(name="layered20k_script", family="layered", pis=100, pos=50, ands=20000, layers=60, window=3, far=0.2,
             from_pis=False, path="resident", commands="b; rw; b; rw -z; b; rw -z; b"),
        # a large flat design, zero-gain replacements allowed
        dict(name="layered1m_rwz_st", family="layered", pis=4096, pos=4096, ands=1000000, layers=200, window=3, far=0.2,
             from_pis=False, path="resident", commands="rw -z; st"),
        # a batch of designs kept on the GPU: the throughput case
        dict(name="batch256_rw_st", family="batch", count=256, lo=1000, hi=200000, min_pis=16, max_pis=512,
             path="resident", commands="rw; st"),
        # many small windows cut out of a larger design
        dict(name="small2000_rw_st", family="batch", count=2000, lo=100, hi=2000, min_pis=8, max_pis=64,
             path="resident", commands="rw; st"),
        # a data set in host arrays, there and back
        dict(name="host100_rw_st", family="batch", count=100, lo=1000, hi=60000, min_pis=16, max_pis=512, path="host",
             commands="rw; st"),
        # a data set as file contents, there and back
        dict(name="aiger128_rw_st", family="batch", count=128, lo=500, hi=100000, min_pis=16, max_pis=512, path="aiger",
             commands="rw; st"),
        # structural hashing alone, as after reading a design
        dict(name="batch128_st", family="batch", count=128, lo=1000, hi=100000, min_pis=16, max_pis=512,
             path="resident", commands="st"),
        # balancing a deep block
        dict(name="mult48_b", family="mult", n=48, path="resident", commands="b"),
        # a burst of jobs on the served mode
        dict(name="served64_rw_st", family="batch", count=64, lo=500, hi=50000, min_pis=16, max_pis=512, path="served",
             commands="rw; st"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["mult", "layered", "layered", "batch", "batch"])
    commands = rng.choice(["rw; st", "rw; st", "rw -z; st", "rw -c; st", "st", "st -c", "b", "b; rw; st",
                           "b; rw; b; rw -z; b"])
    if family == "mult":
        return dict(family="mult", n=_log_uniform(rng, 5, 100), path="resident", commands=commands)
    if family == "layered":
        ands = _log_uniform(rng, 300, 300_000 if "b" in commands else 1_500_000)
        layers = max(4, int(math.sqrt(ands) * math.exp(rng.uniform(-1.6, 0.5))))
        return dict(family="layered", pis=_log_uniform(rng, 8, 3000), pos=_log_uniform(rng, 8, 3000), ands=ands,
                    layers=layers, window=rng.randint(2, 5), far=rng.choice([0.0, 0.0, 0.1, 0.3]),
                    from_pis=rng.random() < 0.5, path=rng.choice(["resident", "host"]), commands=commands)
    path = rng.choice(["resident", "resident", "host", "aiger", "served"])
    if path == "served":
        commands = rng.choice(["rw; st", "rw -z; st"])
    lo = _log_uniform(rng, 60, 3000)
    hi = _log_uniform(rng, 2 * lo, 100 * lo)
    # up to 8M AND nodes in all, 400k where every graph is balanced by itself
    most = max(2, int((400_000 if "b" in commands else 8_000_000) / _mean_size(lo, hi)))
    return dict(family="batch", count=_log_uniform(rng, 2, min(most, 1500)), lo=lo, hi=hi,
                min_pis=rng.randint(4, 16), max_pis=rng.randint(17, 512), path=path, commands=commands)


# ------------------------------------------------------------------ inputs
def _rephased(g, seed, every_fanin):
    """g with other phases: the structure and the sizes are the case's, the
    functions are the seed's.  A multiplier gets some inputs and outputs in
    negative logic; a layered graph's fanin phases are random in any case and
    are drawn again."""
    rng = np.random.default_rng(seed)
    f0, f1, outs = g.fanin0.copy(), g.fanin1.copy(), g.outs.copy()
    a = slice(1 + g.nPIs, None)
    if every_fanin:
        apart = ((f0[a] >> 1) != (f1[a] >> 1)).astype(np.int32)
        f0[a] ^= apart * rng.integers(0, 2, g.nAnds, np.int32)
        f1[a] ^= apart * rng.integers(0, 2, g.nAnds, np.int32)
    else:
        flip = np.zeros(g.nObjs, np.int32)
        flip[1:1 + g.nPIs] = rng.integers(0, 2, g.nPIs)
        f0[a] ^= flip[f0[a] >> 1]
        f1[a] ^= flip[f1[a] >> 1]
        outs ^= flip[outs >> 1]
    outs ^= (outs > 1).astype(np.int32) * rng.integers(0, 2, len(outs), np.int32)
    return C.Aig(g.nPIs, f0, f1, outs)


def _graphs(case, seed):
    if case["family"] == "mult":
        return [_rephased(C.gen_multiplier(case["n"]), seed, False)]
    if case["family"] == "layered":
        graphs = [C.gen_layered(1, case["pis"], case["pos"], case["ands"], case["layers"], case["window"], case["far"],
                                case["from_pis"])]
    else:
        graphs = C.gen_batch(4, 0, case["count"], case["lo"], case["hi"], case["min_pis"], case["max_pis"])
    return [_rephased(g, (seed, i), True) for i, g in enumerate(graphs)]


@functools.cache
def _context():
    return C.Context()


@functools.cache
def _server():
    ctx = C.Context()
    ctx.serve_start(admit_bytes=32 << 30)
    return ctx


@functools.cache
def _library():
    """The C ABI's downloads into buffers that the program keeps."""
    lib = ctypes.CDLL(str(C.LIB_PATH))
    p = ctypes.c_void_p
    lib.culs_batch_download_into.argtypes = [p, p, p, p, p]
    lib.culs_batch_download_aiger_into.argtypes = [p, p, p, ctypes.c_size_t, p]
    return lib


def prepare(case, seed):
    graphs = _graphs(case, seed)
    state = dict(path=case["path"], commands=[c.strip() for c in case["commands"].split(";")])
    n, n_po = sum(g.nObjs for g in graphs), sum(g.nPOs for g in graphs)
    # where the results go: no command makes a graph much larger
    state["fanins"] = [np.zeros(n + n // 4 + 64, np.int32) for _ in range(2)]
    state["outs"] = np.zeros(n_po, np.int32)
    state["levels"] = np.zeros(len(graphs), np.int32)
    if case["path"] == "served":
        state.update(ctx=_server(), graphs=graphs)
        return state
    ctx = state["ctx"] = _context()
    if case["path"] == "resident":
        state["input"] = ctx.upload_batch(graphs) if len(graphs) > 1 else ctx.upload(graphs[0])
        state["work"] = ctx.clone(state["input"])
    elif case["path"] == "aiger":
        state["files"] = [bytes(f) for f in ctx.upload_batch(graphs).download_aiger_all()]
        state["bytes"] = np.zeros(10 * n + 12 * n_po + 1024 * len(graphs), np.uint8)
        state["offsets"] = np.zeros(len(graphs) + 1, np.uint64)
    else:
        state["graphs"] = graphs
    return state


# -------------------------------------------------------------------- pass
def _execute(ctx, d, commands):
    k = 0
    while k < len(commands):
        c = commands[k]
        if c.startswith("rw") and commands[k + 1:k + 2] and commands[k + 1].startswith("st"):
            ctx.rw_st(d, zeros="-z" in c, gpu_dedup="-c" not in c, cpu_st="-c" in commands[k + 1])
            k += 2
            continue
        if c.startswith("rw"):
            ctx.rw(d, zeros="-z" in c, gpu_dedup="-c" not in c)
        elif c.startswith("st"):
            ctx.st(d, cpu="-c" in c)
        else:
            ctx.b(d)
        k += 1


def _starts(sizes):
    starts = np.zeros(len(sizes) + 1, np.int64)
    np.cumsum(sizes, out=starts[1:])
    return starts


def _download(state, d):
    """Every graph's arrays, back to back in the state's buffers."""
    s = d.stats_all()
    objs, outs = _starts(1 + s["nPIs"].astype(np.int64) + s["nAnds"]), _starts(s["nPOs"].astype(np.int64))
    if objs[-1] > len(state["fanins"][0]):
        raise RuntimeError("the result is larger than the kept buffers")
    at = [np.ascontiguousarray(b.ctypes.data + 4 * o[:-1], dtype=np.uint64)
          for b, o in ((state["fanins"][0], objs), (state["fanins"][1], objs), (state["outs"], outs))]
    if _library().culs_batch_download_into(state["ctx"].h, d.h, *[a.ctypes.data for a in at]):
        raise RuntimeError("download failed")
    return dict(ands=s["nAnds"], levels=s["nLevels"], fanins=state["fanins"], outs=state["outs"])


def _serve(state):
    ctx, at, po = state["ctx"], 0, 0
    jobs = [ctx.submit(g, zeros="rw -z" in state["commands"]) for g in state["graphs"]]
    for i, j in enumerate(jobs):
        ctx.wait(j)
        g, _ = ctx.fetch(j)
        for kept, a in zip(state["fanins"], (g.fanin0, g.fanin1)):
            kept[at:at + g.nObjs] = a
        state["outs"][po:po + g.nPOs] = g.outs
        state["levels"][i] = g.nLevels
        at, po = at + g.nObjs, po + g.nPOs
    return dict(levels=state["levels"], fanins=state["fanins"], outs=state["outs"])


def run(state):
    ctx, commands, path = state["ctx"], state["commands"], state["path"]
    if path == "served":
        return _serve(state)
    if path == "aiger":
        d = ctx.upload_aiger_batch(state["files"])
        _execute(ctx, d, commands)
        if _library().culs_batch_download_aiger_into(ctx.h, d.h, state["bytes"].ctypes.data, state["bytes"].size,
                                                     state["offsets"].ctypes.data):
            raise RuntimeError("download failed")
        return dict(levels=d.stats_all()["nLevels"], files=state["bytes"], offsets=state["offsets"].astype(np.int64))
    if path == "host":
        graphs = state["graphs"]
        d = ctx.upload_batch(graphs) if len(graphs) > 1 else ctx.upload(graphs[0])
    else:
        d = ctx.clone(state["input"], into=state["work"])
    _execute(ctx, d, commands)
    return _download(state, d)


# ---------------------------------------------------------------- measures
def _mean_size(lo, hi):
    return (hi - lo) / math.log(hi / lo) if hi > lo else lo


def work(case):
    """Two 32-bit fanin literals of every AND node, read once and written
    once (the results are nearly as large as the inputs); the commands need no
    floating-point operations."""
    if case["family"] == "mult":
        ands = 10 * case["n"] ** 2
    elif case["family"] == "layered":
        ands = case["ands"]
    else:
        ands = case["count"] * _mean_size(case["lo"], case["hi"])
    return {"bytes": 16.0 * ands, "flops": 0.0}


def tolerance(case):
    return "exact"
