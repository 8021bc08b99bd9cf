"""The work a user of this framework has it do, as cases that can be timed.

Most cases are whole builds of the all-points kNN graph (`Context.build`, what
the command line and the Python front end call), from the smallest jobs of the
tests and of the batched mix to the largest of the serving mix; the others are a
batch of mixed jobs and single stages through their own entry points.  Rows are
the seeded Gaussian mixtures of `synth` (unit rows, Zipf cluster sizes, one
centre per hundred rows as in the benchmark's configurations) or rows of a
random 64-dimensional subspace, where the graph reaches the recall it has on
real embeddings.

    listed()  draw(rng)  prepare(case, seed)  run(state)  work(case)  exact(case, seed)
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sisap-2026-task1_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import knng  # noqa: E402
import synth  # noqa: E402

DIMS = (128, 256, 384, 512, 640, 768, 896, 1024)
K_BUILD, K_EVAL, TREES, LEAF, RERANK = 50, 15, 16, 64, 400


def listed():
    return [
        # the smallest job: a few thousand rows (the size of the test fixtures, below the
        # smallest job of the batched mix), where launches and waits are most of the time
        {"name": "build_2k_384", "kind": "build", "n": 2003, "d": 384, "data": "mixture", "rows": "device"},
        # an ordinary small job of the serving mix (10k to 2M rows), a ragged number of rows
        {"name": "build_20k_768", "kind": "build", "n": 20011, "d": 768, "data": "mixture", "rows": "device"},
        # the plain small configuration of the benchmark
        {"name": "build_100k_1024", "kind": "build", "n": 100000, "d": 1024, "data": "mixture", "rows": "device"},
        # rows of low intrinsic dimension, like the spectrum of real embeddings: the graph
        # converges to high recall and rows share few candidates by chance
        {"name": "build_300k_subspace", "kind": "build", "n": 300000, "d": 1024, "data": "subspace", "rows": "device"},
        # the largest jobs of the serving mix, on the way to the 6.35M rows of the contest
        {"name": "build_2m_1024", "kind": "build", "n": 2000000, "d": 1024, "data": "mixture", "rows": "device"},
        # the command line's and numpy users' way in: pageable host rows in, host graph out
        {"name": "build_200k_384_numpy", "kind": "build", "n": 200003, "d": 384, "data": "mixture", "rows": "numpy"},
        # the optional 128-bit hyperplane sketch
        {"name": "build_150k_512_hyperplane", "kind": "build", "n": 150001, "d": 512, "data": "mixture",
         "rows": "device", "sketch": "hyperplane"},
        # independent jobs of several dimensions built together, as the serving loop does
        {"name": "batch_24_jobs", "kind": "batch", "jobs": 24, "lo": 5000, "hi": 200000, "pick": 7},
        # the stages by themselves: int8 codes and sign sketches of new rows
        {"name": "quantize_1m_1024", "kind": "quantize", "n": 1000000, "d": 1024, "mode": "trunc"},
        # the random-projection forest of 16 trees
        {"name": "forest_500k_768", "kind": "forest", "n": 500009, "d": 768},
        # the initial graph from the forest's leaves
        {"name": "init_graph_200k_896", "kind": "init_graph", "n": 200001, "d": 896},
        # one NN-Descent iteration on a graph of the caller's
        {"name": "join_iter_100k_1024", "kind": "join_iter", "n": 100003, "d": 1024},
    ]


def _spread(rng, lo, hi):
    """Log-uniform whole number, odd sizes among them."""
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(("build", "build", "build", "build", "build", "batch", "quantize", "forest", "init_graph",
                       "join_iter"))
    d = rng.choice(DIMS)
    if kind == "build":
        case = {"kind": kind, "n": _spread(rng, 2000, 1000000), "d": d,
                "data": rng.choice(("mixture", "mixture", "mixture", "subspace")),
                "rows": rng.choice(("device", "device", "numpy"))}
        if rng.random() < 0.2:
            case["sketch"] = "hyperplane"
        return case
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 32), "lo": 5000, "hi": _spread(rng, 10000, 200000),
                "pick": rng.randrange(1 << 20)}
    if kind == "quantize":
        return {"kind": kind, "n": _spread(rng, 2000, 2000000), "d": d, "mode": rng.choice(("trunc", "round"))}
    return {"kind": kind, "n": _spread(rng, 2000, 1000000), "d": d}


def _rows(n, d, data, seed):
    """(n, d) float32 unit rows on the GPU."""
    if data == "mixture":
        return synth.mixture_torch(n, d, max(10, n // 100), seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    basis = torch.randn(64, d, generator=g, device="cuda")
    x = torch.empty(n, d, device="cuda")
    for s in range(0, n, 1 << 18):
        e = min(n, s + (1 << 18))
        y = torch.randn(e - s, 64, generator=g, device="cuda") @ basis
        x[s:e] = y / y.norm(dim=1, keepdim=True)
    return x


def _batch_shapes(case):
    """The (n, d) of a batch's jobs: sizes log-uniform, dimensions of the benchmark's mix."""
    rng = np.random.Generator(np.random.PCG64(case["pick"]))
    n = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["jobs"])).astype(int)
    d = rng.choice((384, 768, 1024), case["jobs"])
    return [(int(a), int(b)) for a, b in zip(n, d)]


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "batch":
        s["ctx"] = knng.Context()
        s["rows"] = [_rows(n, d, "mixture", 1000 * seed + b) for b, (n, d) in enumerate(_batch_shapes(case))]
        return s
    if kind == "build":
        x = _rows(case["n"], case["d"], case["data"], seed)
        s["rows"] = x.cpu().numpy() if case["rows"] == "numpy" else x
        hyper = case.get("sketch") == "hyperplane"
        s["ctx"] = knng.Context(sketch_mode=knng.SKETCH_HYPERPLANE if hyper else knng.SKETCH_SIGN)
        return s
    x = _rows(case["n"], case["d"], "mixture", seed)
    if kind == "quantize":
        s["rows"] = x
        s["mode"] = knng.QUANT_ROUND if case["mode"] == "round" else knng.QUANT_TRUNC
        return s
    s["codes"], s["sketch"] = knng.quantize(x)
    s["ctx"] = knng.Context()
    if kind in ("init_graph", "join_iter"):
        s["perm"], s["leaf"] = s["ctx"].forest(s["codes"])
    if kind == "join_iter":
        s["ids"], s["scores"] = s["ctx"].init_graph(s["codes"], s["perm"], s["leaf"])
    return s


def run(s):
    kind = s["kind"]
    if kind == "build":
        knns, dists, stats = s["ctx"].build(s["rows"])
        return {"knns": knns, "dists": dists, "iterations": stats.iterations}
    if kind == "batch":
        out, _ = s["ctx"].build_batch(s["rows"])
        return {"knns": torch.cat([k for k, _, _ in out]), "dists": torch.cat([v for _, v, _ in out]),
                "iterations": [int(i) for _, _, i in out]}
    if kind == "quantize":
        codes, sketch = knng.quantize(s["rows"], s["mode"])
        return {"codes": codes, "sketch": sketch}
    if kind == "forest":
        perm, leaf = s["ctx"].forest(s["codes"])
        return {"perm": perm, "leaf_flag": leaf}
    if kind == "init_graph":
        ids, scores = s["ctx"].init_graph(s["codes"], s["perm"], s["leaf"])
        return {"ids": ids, "scores": scores}
    ids, scores, updates = s["ctx"].join_iter(s["codes"], s["sketch"], s["ids"], s["scores"])
    return {"ids": ids, "scores": scores, "updates": updates}


def _forest_flops(n, d):
    # two dots of d products per member and level, in every tree
    return TREES * max(1.0, math.log2(max(2.0, n / (0.7 * LEAF)))) * n * 2 * d * 2


def _init_flops(n, d):
    return TREES * n * 0.7 * LEAF / 2 * d * 2  # every pair of a leaf once, leaves 70 % full


def _join_flops(n, d):
    return n * RERANK * d * 2  # the reranked candidates' dots of one iteration


def work(case):
    """Each input read once, each output written once; the operations that the algorithm's definition counts."""
    kind = case["kind"]
    if kind in ("build", "batch"):
        shapes = _batch_shapes(case) if kind == "batch" else [(case["n"], case["d"])]
        return {"bytes": sum(n * d * 4 + n * K_EVAL * 8 for n, d in shapes),
                "flops": sum(_forest_flops(n, d) + _init_flops(n, d) + 2 * _join_flops(n, d) for n, d in shapes)}
    n, d = case["n"], case["d"]
    if kind == "quantize":
        return {"bytes": n * d * 4 + n * d + n * d / 8, "flops": n * d * 2}
    if kind == "forest":
        return {"bytes": n * d + TREES * n * 5, "flops": _forest_flops(n, d)}
    if kind == "init_graph":
        return {"bytes": n * d + TREES * n * 5 + n * K_BUILD * 8, "flops": _init_flops(n, d)}
    return {"bytes": n * d + n * d / 8 + 2 * n * K_BUILD * 8, "flops": _join_flops(n, d)}


def exact(case, seed):
    """None: every output is a whole number (the distances of a graph are the int8 inner products of
    the neighbours that the build settles on), which other arithmetic cannot come nearer to."""
    return None
