"""The join's duplicate search (tagged atomic-min tables) at the edges of its range.

The kernel has a compile-time form for K = 50, R = 400 on 8-byte aligned lists
and a general form for everything else.  Both are compared bit for bit with the
oracle's iteration (src/main.cpp:324-430, double-buffered, stable ties):

* list lengths at the edges of the pair layout (odd K, one occurrence, K = 64
  with 8 pairs per thread), more and fewer candidates than the rerank set,
  and few rows, where almost every candidate repeats and ids lose several
  table rounds;
* lists that start on a 4-byte boundary only;
* whole builds with the candidate cache, whose cached ids are looked up in the
  same rounds, against builds without it.
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


def _stable(**kw):
    return oracle.params(threads=os.cpu_count() or 1, tie_mode=oracle.TIE_STABLE, jacobi=1, **kw)


def _at_offset(torch, a, offset):
    """A CUDA copy of int32 array `a` that starts `offset` elements into its storage."""
    buf = torch.zeros(a.size + offset, dtype=torch.int32, device="cuda")
    buf[offset:] = torch.from_numpy(np.ascontiguousarray(a).reshape(-1)).cuda()
    return buf[offset:].view(a.shape)


@pytest.mark.parametrize("k,mult,n,d,offset", [
    (50, 8, 1500, 1024, 0), (50, 8, 1500, 384, 1), (50, 8, 90, 128, 0), (50, 7, 1500, 256, 0), (50, 80, 800, 128, 0),
    (1, 8, 700, 128, 0), (2, 1, 700, 128, 0), (3, 4, 900, 640, 1), (49, 8, 1500, 256, 0), (51, 8, 1500, 128, 0),
    (64, 8, 2500, 896, 0), (64, 64, 300, 128, 0),
])
def test_iterations_bit_exact(env, k, mult, n, d, offset):
    torch, knng = env
    x = synth.mixture(n, d, max(5, n // 60), seed=1000 + n + k)
    codes_h, sk_h = oracle.quantize(x)
    prm = _stable(k_build=k, k_eval=min(15, k), rerank_mult=mult)
    perm, lf, _ = oracle.forest(codes_h, prm)
    ids_ref, sc_ref = oracle.init_graph(codes_h, perm, lf, prm)
    ids = _at_offset(torch, ids_ref, offset)
    sc = _at_offset(torch, sc_ref, offset)
    codes = torch.from_numpy(codes_h).cuda()
    sk = torch.from_numpy(sk_h.view(np.int64)).cuda()
    with knng.Context(k_build=k, k_eval=min(15, k), rerank_mult=mult) as ctx:
        for it in range(3):
            up_ref = oracle.join_iter(codes_h, sk_h, ids_ref, sc_ref, prm)
            out_ids, out_sc = _at_offset(torch, np.zeros_like(ids_ref), offset), _at_offset(torch, np.zeros_like(sc_ref), offset)
            ids, sc, up = ctx.join_iter(codes, sk, ids, sc, out_ids, out_sc)
            assert up == up_ref, f"iteration {it}"
            np.testing.assert_array_equal(ids.cpu().numpy(), ids_ref)
            np.testing.assert_array_equal(sc.cpu().numpy(), sc_ref)


@pytest.mark.parametrize("k,mult,n,d,sketch", [
    (50, 8, 9000, 768, 0), (50, 8, 4000, 128, 1), (33, 8, 6000, 512, 0), (64, 8, 6000, 256, 1), (15, 20, 5000, 384, 0),
])
def test_build_with_cache_equals_build_without(env, k, mult, n, d, sketch):
    torch, knng = env
    x = torch.from_numpy(synth.subspace(n, d, 24, seed=n + k)).cuda()
    got = []
    for cache in (0, 1):
        with knng.Context(k_build=k, rerank_mult=mult, join_cache=cache, sketch_mode=sketch) as ctx:
            st = knng.Stats()
            knns, dists, _ = ctx.build(x, stats=st)
        got.append((knns.cpu().numpy(), dists.cpu().numpy(), st.iterations, list(st.updates[: st.iterations]),
                    list(st.join_distinct[: st.iterations])))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    assert got[0][2:] == got[1][2:] and got[0][2] >= 2
