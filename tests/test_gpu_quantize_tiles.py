"""The quantise kernel at the edges of its blocks (512 groups of 8 floats) and
warps (32 groups a step), bit for bit against the oracle's restatement of
src/main.cpp:179-192, with rows that start 16 bytes into an allocation."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(1, 64), (3, 64), (5, 64), (63, 64), (64, 64), (65, 64), (1, 1024), (21, 192), (33, 128)])
@pytest.mark.parametrize("mode", [oracle.QUANT_TRUNC, oracle.QUANT_ROUND])
def test_quantize_block_edges(n, d, mode):
    import torch

    import knng

    rng = np.random.default_rng(n * d)
    x = (rng.standard_normal((n, d)) * 0.7).astype(np.float32)
    x[:, ::7] = np.array([np.nan, np.inf, -np.inf, 1e-40, -0.0, 0.5 / 127, -128.6 / 127], np.float32)[
        rng.integers(0, 7, size=x[:, ::7].shape)]
    codes_ref, sk_ref = oracle.quantize(x, mode)
    buf = torch.empty(n * d + 4, dtype=torch.float32, device="cuda")
    rows = buf[4:].view(n, d)
    rows.copy_(torch.from_numpy(x))
    codes, sk = knng.quantize(rows, mode)
    np.testing.assert_array_equal(codes.cpu().numpy(), codes_ref)
    np.testing.assert_array_equal(sk.cpu().numpy().view(np.uint64), sk_ref)
