"""The initial graph's selection and leaf Grams at the edges of their ranges.

Against the oracle's initial graph on the same forest (best K distinct by score
desc, id asc; src/main.cpp:234-314):

* equal scores everywhere (identical rows, a handful of distinct rows): more
  ties at the K-th place than are ranked, so the selection descends into ids;
* more trees than one group of candidates holds, one tree, few candidates;
* K = 1 and K = 64; leaves of every size from 1 to 64 members (the Gram has one
  body per 8 members), extreme codes whose dots reach 2^24.
"""
import os

import numpy as np
import pytest

import oracle
import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch

    assert torch.cuda.is_available(), "the gpu tests need a CUDA device"
    import knng

    knng.lib()
    return torch, knng


def _codes(kind, n, d):
    rng = np.random.default_rng(n + d)
    if kind == "same":
        return np.full((n, d), 5, np.int8)
    if kind == "few":
        return rng.integers(-30, 30, (3, d)).astype(np.int8)[np.arange(n) % 3]
    if kind == "extreme":
        return rng.choice(np.array([-128, 127, -127, 126, 1], np.int8), (n, d), p=[0.6, 0.25, 0.05, 0.05, 0.05])
    return oracle.quantize(synth.mixture(n, d, max(3, n // 90), seed=n + d))[0]


@pytest.mark.parametrize("kind,n,d,leaf,trees,k", [
    ("same", 900, 128, 64, 16, 50), ("few", 1500, 128, 64, 16, 50), ("few", 1500, 256, 64, 40, 64),
    ("extreme", 1200, 1024, 64, 16, 50), ("mix", 2500, 640, 64, 33, 64), ("mix", 2500, 384, 64, 1, 50),
    ("mix", 3000, 896, 37, 20, 1), ("mix", 70, 128, 64, 16, 50), ("mix", 2000, 512, 9, 64, 50),
    ("same", 300, 128, 64, 64, 64),
])
def test_init_graph_equals_oracle(env, kind, n, d, leaf, trees, k):
    torch, knng = env
    codes_h = _codes(kind, n, d)
    codes = torch.from_numpy(codes_h).cuda()
    prm = oracle.params(threads=os.cpu_count() or 1, tie_mode=oracle.TIE_STABLE, jacobi=1, k_build=k,
                        k_eval=min(15, k), leaf_size=leaf, num_trees=trees)
    perm, lf, _ = oracle.forest(codes_h, prm)
    ids_ref, sc_ref = oracle.init_graph(codes_h, perm, lf, prm)
    with knng.Context(k_build=k, k_eval=min(15, k), leaf_size=leaf, num_trees=trees) as ctx:
        ids, sc = ctx.init_graph(codes, torch.from_numpy(perm).cuda(), torch.from_numpy(lf).cuda())
    np.testing.assert_array_equal(sc.cpu().numpy(), sc_ref)
    np.testing.assert_array_equal(ids.cpu().numpy(), ids_ref)


@pytest.mark.parametrize("d", [128, 1024])
def test_leaves_of_every_size(env, d):
    torch, knng = env
    sizes = np.concatenate([np.arange(1, 65), np.arange(64, 0, -1), [64] * 10])
    n = int(sizes.sum())
    rng = np.random.default_rng(d)
    codes_h = _codes("extreme", n, d)
    perm = np.stack([rng.permutation(n) for _ in range(3)]).astype(np.int32)
    lf = np.zeros((3, n), np.uint8)
    for t in range(3):
        rng.shuffle(sizes)
        lf[t, np.concatenate([[0], np.cumsum(sizes)[:-1]])] = 1
    prm = oracle.params(threads=1, tie_mode=oracle.TIE_STABLE, jacobi=1, num_trees=3)
    ids_ref, sc_ref = oracle.init_graph(codes_h, perm, lf, prm)
    with knng.Context(num_trees=3) as ctx:
        ids, sc = ctx.init_graph(torch.from_numpy(codes_h).cuda(), torch.from_numpy(perm).cuda(),
                                 torch.from_numpy(lf).cuda())
    np.testing.assert_array_equal(sc.cpu().numpy(), sc_ref)
    np.testing.assert_array_equal(ids.cpu().numpy(), ids_ref)
