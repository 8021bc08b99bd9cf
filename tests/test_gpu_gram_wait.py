"""Results of the leaf Gram's tcgen05 form, which a positive wait_limit selects.

The default form (warp-level tensor-core instructions) has no device wait; a
caller who bounds the waits gets the tcgen05 kernel, whose waits honour the
limit.  With a limit that is never reached the initial graph must equal the
oracle's, and a build must equal the default form's, bit for bit.
"""
import numpy as np
import pytest

import oracle
import synth
from test_gpu_gram_tc import _extreme_rows

pytestmark = pytest.mark.gpu
LIMIT = 1 << 26  # the default number of polls


@pytest.mark.parametrize("n,d,leaf,kind", [(3000, 1024, 64, "mix"), (5000, 384, 64, "mix"), (2500, 768, 17, "mix"),
                                           (700, 1024, 64, "extreme"), (900, 128, 64, "extreme"), (37, 1024, 64, "mix")])
def test_init_graph_with_a_wait_limit_is_bit_exact(n, d, leaf, kind):
    import torch

    import knng

    x = synth.mixture(n, d, max(1, n // 100), seed=n + d) if kind == "mix" else _extreme_rows(n, d, n)
    codes_ref, _ = oracle.quantize(x)
    prm = oracle.params(threads=1, tie_mode=oracle.TIE_STABLE, jacobi=1, leaf_size=leaf)
    perm_ref, lf_ref, _ = oracle.forest(codes_ref, prm)
    ids_ref, sc_ref = oracle.init_graph(codes_ref, perm_ref, lf_ref, prm)
    codes, perm, lf = (torch.from_numpy(a).cuda() for a in (codes_ref, perm_ref, lf_ref))
    for limit in (LIMIT, 0):
        with knng.Context(gram_mode=knng.GRAM_TCGEN05, wait_limit=limit, leaf_size=leaf) as ctx:
            ids, sc = ctx.init_graph(codes, perm, lf)
        np.testing.assert_array_equal(sc.cpu().numpy(), sc_ref, err_msg=f"wait_limit {limit}")
        np.testing.assert_array_equal(ids.cpu().numpy(), ids_ref, err_msg=f"wait_limit {limit}")


def test_build_with_a_wait_limit_equals_the_default():
    import knng

    x = synth.mixture(30000, 1024, 300, seed=77)
    got = []
    for limit in (0, LIMIT):
        with knng.Context(gram_mode=knng.GRAM_TCGEN05, wait_limit=limit) as ctx:
            got.append(ctx.build(x))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    assert got[0][2].iterations == got[1][2].iterations
