"""The native forest at its limits: the depth valve beside ordinary rows.

Thousands of equal rows lose three members per fused round, so the rounds go on
until the depth valve (2048 levels, csrc/forest.cu) cuts what is left of them
into consecutive leaves.  The valve belongs to the node that reached its depth:
the other nodes of the same forest, and the other jobs of the same batch, are
split as they are without those rows.
"""
import numpy as np
import pytest

import synth
from test_gpu_forest_native import _fused_pivots, _mix, _node_hash, _sides

pytestmark = pytest.mark.gpu
VALVE = 2048  # levels, csrc/forest.cu


def forest_with_valve(codes, trees, leaf, seed):
    """csrc/forest.cu's rules with a depth per node: a fused round takes three levels, a node of
    fewer than 512 members is split one level at a time from the depth at which its round ended."""
    n = len(codes)
    codes = codes.astype(np.int64)
    perm, flags, valves = np.tile(np.arange(n), (trees, 1)), np.zeros((trees, n), np.uint8), 0
    for t in range(trees):
        row = perm[t]
        todo = [(0, n, True, 0)]
        while todo:
            s, size, fused, depth = todo.pop()
            if size <= leaf:
                flags[t, s] = 1
                continue
            if depth >= VALVE:
                flags[t, s:s + size:leaf] = 1
                valves += 1
                continue
            seg, h = row[s:s + size].copy(), _node_hash(seed, t, s, size)
            if not fused:
                a, b = h % size, _mix(h ^ 0x5851F42D4C957F2D) % (size - 1)
                side = _sides(codes, seg, seg[a], seg[b + (b >= a)])
                row[s:s + size] = np.concatenate([seg[side == 0], seg[side == 1]])
                nl = int((side == 0).sum())
                todo += [(s, nl, False, depth + 1), (s + nl, size - nl, False, depth + 1)]
                continue
            piv = _fused_pivots(codes, seg, h)
            ends = []  # (first path code, one past the last) of the descendants that the round leaves

            def walk(q, members, level, lo, hi, code):
                if q not in piv:
                    ends.append((lo, hi))
                    return
                bit = _sides(codes, seg[members], *piv[q])
                code[members] |= bit << (2 - level)
                mid = (lo + hi) // 2
                for b, (clo, chi) in enumerate(((lo, mid), (mid, hi))):
                    sub = members[bit == b]
                    if level < 2 and len(sub) > leaf:
                        walk(2 * q + 1 + b, sub, level + 1, clo, chi, code)
                    else:
                        ends.append((clo, chi))
                        if level < 2:  # a leaf: its members still sort by the deeper splits
                            _deeper(codes, seg, piv, 2 * q + 1 + b, sub, level + 1, code)

            code = np.zeros(size, int)
            walk(0, np.arange(size), 0, 0, 8, code)
            row[s:s + size] = seg[np.argsort(code, kind="stable")]
            pre = np.concatenate([[0], np.cumsum(np.bincount(code, minlength=8))])
            for lo, hi in ends:
                c = int(pre[hi] - pre[lo])
                todo.append((s + int(pre[lo]), c, c >= 512, depth + 3))
    return perm, flags, valves


def _deeper(codes, seg, piv, q, members, level, code):
    if q not in piv or level > 2 or not len(members):
        return
    bit = _sides(codes, seg[members], *piv[q])
    code[members] |= bit << (2 - level)
    for b in (0, 1):
        _deeper(codes, seg, piv, 2 * q + 1 + b, members[bit == b], level + 1, code)


def _mixture_codes(n, d, seed):
    return np.trunc(synth.mixture(n, d, max(3, n // 80), seed=seed) * 127).astype(np.int8)


@pytest.fixture(scope="module")
def env():
    import torch

    assert torch.cuda.is_available(), "the gpu tests need a CUDA device"
    import knng

    knng.lib()
    return torch, knng


def test_valve_of_equal_rows_leaves_other_nodes_alone(env):
    torch, knng = env
    codes = np.concatenate([np.full((3600, 128), 3, np.int8), _mixture_codes(3000, 128, 11)])
    codes = codes[np.random.default_rng(5).permutation(len(codes))]
    ref_perm, ref_flags, valves = forest_with_valve(codes, 2, 64, 1337)
    assert valves >= 2  # each tree's equal rows reach it
    with knng.Context(num_trees=2) as ctx:
        perm, flags = ctx.forest(torch.from_numpy(codes).cuda())
    np.testing.assert_array_equal(perm.cpu().numpy(), ref_perm)
    np.testing.assert_array_equal(flags.cpu().numpy(), ref_flags)


def test_batched_job_beside_equal_rows_equals_its_solo_build(env):
    torch, knng = env
    same = np.tile(synth.mixture(1, 256, 1, seed=3), (4000, 1))
    other = synth.mixture(7000, 256, 70, seed=4)
    with knng.Context() as ctx:
        solo = [ctx.build(x) for x in (same, other)]
    with knng.Context() as ctx:
        res, _ = ctx.build_batch([np.ascontiguousarray(same), other])
    for (k, dd, it), (ks, ds, st) in zip(res, solo):
        np.testing.assert_array_equal(k, ks)
        np.testing.assert_array_equal(dd, ds)
        assert it == st.iterations


def _extreme_codes(n, d, kind, seed):
    rng = np.random.default_rng(seed)
    if kind == "ends":  # dots up to d * 2^14 either way
        codes = rng.choice(np.array([-128, 127, -1, 0, 1], np.int8), size=(n, d))
        codes[: n // 8], codes[n // 8: n // 4] = -128, 127
    else:  # dots of 0.99 * d * 2^14, a few units apart
        codes = np.where(rng.random((n, d)) < 0.5, -127, -128).astype(np.int8)
    return codes[rng.permutation(n)]


@pytest.mark.parametrize("n,d,kind", [(3001, 1024, "ends"), (3001, 1024, "near"), (2000, 128, "ends"), (1300, 640, "near")])
def test_forest_of_extreme_codes(env, n, d, kind):
    """The member pass takes its dots in f16 with fp32 sums: exact up to 2^24, which 1024 codes of -128 reach."""
    torch, knng = env
    codes = _extreme_codes(n, d, kind, n + d)
    ref_perm, ref_flags, _ = forest_with_valve(codes, 2, 64, 1337)
    with knng.Context(num_trees=2) as ctx:
        perm, flags = ctx.forest(torch.from_numpy(codes).cuda())
    np.testing.assert_array_equal(perm.cpu().numpy(), ref_perm)
    np.testing.assert_array_equal(flags.cpu().numpy(), ref_flags)
