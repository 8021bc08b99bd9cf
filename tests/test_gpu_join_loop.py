"""The NN-Descent phase as a graph loop equals the iterations launched one by one.

Iterations 0 and 1 are straight graph nodes, 2 and 3 the body of a loop node:
every small limit ends at another place of that structure (before the loop, in
the middle of a body, at its end), and so does the early stop.  The in-place
mode is left out: its rows race by design.
"""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [0, 1, 2, 3, 4, 5, 30])
def test_loop_equals_single_launches(limit):
    import torch

    assert torch.cuda.is_available(), "the gpu tests need a CUDA device"
    import knng

    x = torch.from_numpy(synth.mixture(20000, 256, 200, seed=9)).cuda()
    small = torch.from_numpy(synth.mixture(700, 256, 7, seed=10)).cuda()  # stops before the other
    got = []
    for graph in (1, 0):
        with knng.Context(max_iterations=limit, use_graph=graph) as ctx:
            for _ in range(2):  # captured, then replayed
                st = knng.Stats()
                knns, dists, _ = ctx.build(x, stats=st)
            out, _ = ctx.build_batch([x, small])
        ms = list(st.join_ms[: st.iterations])
        assert all(0.0 < t < 1000.0 for t in ms)
        got.append((st.iterations, list(st.updates[: st.iterations]), knns.cpu().numpy(), dists.cpu().numpy(),
                    [i for _, _, i in out], out[0][0].cpu().numpy(), out[1][0].cpu().numpy()))
    assert got[0][:2] == got[1][:2] and got[0][4] == got[1][4]
    assert got[0][0] == min(limit, got[0][0]) and got[0][4][0] == got[0][0]
    if limit == 30:
        assert got[0][4][1] < got[0][4][0] > 2
    for q in (2, 3, 5, 6):
        np.testing.assert_array_equal(got[0][q], got[1][q])
    np.testing.assert_array_equal(got[0][2], got[0][5])
