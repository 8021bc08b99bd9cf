"""The native forest (fused rounds, then one kernel per small subtree) against numpy.

The numpy restatement follows the rules stated in csrc/forest.cu: the hashed
node identity (seed, tree, local start, size), three levels per pass from a
sample of 64 members for roots and nodes of at least 512 members, one level at
a time below, stable splits by exact integer dots.  The permutation and the
leaf flags must be equal, at sizes around the 512-member line, for small and
odd leaf sizes (many open descendants per subtree, beyond the staged pivot
rows), duplicated rows (splits that peel off one member per level) and batches'
several jobs per tree.
"""
import math

import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu
M64 = (1 << 64) - 1


def _mix(x):
    x = (x + 0x9E3779B97F4A7C15) & M64
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & M64
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & M64
    return x ^ (x >> 31)


def _node_hash(seed, tree, local, size):
    return _mix(_mix(_mix((seed << 32) ^ tree) ^ local) ^ (size << 1))


def _sides(codes, ids, p1, p2):
    d = codes[ids] @ np.stack([codes[p1], codes[p2]], axis=1)
    side = np.where(d[:, 0] > d[:, 1], 0, 1)
    side[ids == p1] = 0
    side[ids == p2] = 1
    return side


def _fused_pivots(codes, seg, h):
    size = len(seg)
    a, b = h % size, 1 + _mix(h ^ 0x2545F4914F6CDD1D) % (size - 1)
    while math.gcd(b, size) != 1:
        b = 1 if b + 1 == size else b + 1
    cand = seg[[(a + q * b) % size for q in range(min(size, 64))]]
    node, used, piv = np.zeros(len(cand), int), np.zeros(len(cand), bool), {}
    for depth in range(3):
        for j in range((1 << depth) - 1, (2 << depth) - 1):
            free = np.flatnonzero((node == j) & ~used)
            if len(free) >= 2:
                piv[j] = (cand[free[0]], cand[free[1]])
                used[free[:2]] = True
        if depth == 2:
            return piv
        new = np.full(len(cand), -1)
        for j in piv:
            at = np.flatnonzero(node == j)
            if len(at):
                new[at] = 2 * j + 1 + _sides(codes, cand[at], *piv[j])
        node = new
    return piv


def native_forest(codes, trees, leaf, seed):
    n = len(codes)
    codes = codes.astype(np.int64)
    perm = np.tile(np.arange(n), (trees, 1))
    flags = np.zeros((trees, n), np.uint8)
    for t in range(trees):
        row = perm[t]
        todo = [(0, n, True)] if n > leaf else []
        if n <= leaf:
            flags[t, 0] = 1
        while todo:
            s, size, fused = todo.pop()
            seg, h = row[s:s + size].copy(), _node_hash(seed, t, s, size)
            if not fused:
                a, b = h % size, _mix(h ^ 0x5851F42D4C957F2D) % (size - 1)
                b += b >= a
                side = _sides(codes, seg, seg[a], seg[b])
                row[s:s + size] = np.concatenate([seg[side == 0], seg[side == 1]])
                nl = int((side == 0).sum())
                kids = [(s, nl), (s + nl, size - nl)]
            else:
                piv = _fused_pivots(codes, seg, h)
                code, j, live = np.zeros(size, int), np.zeros(size, int), np.ones(size, bool)
                for depth in range(3):
                    nj = j.copy()
                    for q in range((1 << depth) - 1, (2 << depth) - 1):
                        at = np.flatnonzero(live & (j == q))
                        if q in piv and len(at):
                            bit = _sides(codes, seg[at], *piv[q])
                            code[at] |= bit << (2 - depth)
                            nj[at] = 2 * q + 1 + bit
                        else:
                            live[at] = False
                    j = nj
                row[s:s + size] = seg[np.argsort(code, kind="stable")]
                count = np.bincount(code, minlength=8)
                pre = np.concatenate([[0], np.cumsum(count)])
                kids, split = [], [0]
                while split:
                    q = split.pop()
                    depth = (q + 1).bit_length()
                    for ch in (2 * q + 1, 2 * q + 2):
                        p = ch - ((1 << depth) - 1)
                        lo, hi = pre[p << (3 - depth)], pre[(p + 1) << (3 - depth)]
                        if hi - lo > leaf and depth < 3 and ch in piv:
                            split.append(ch)
                        else:
                            kids.append((s + int(lo), int(hi - lo)))
            for cs, csize in kids:
                assert csize > 0
                if csize <= leaf:
                    flags[t, cs] = 1
                else:
                    todo.append((cs, csize, csize >= 512))
    return perm, flags


@pytest.fixture(scope="module")
def env():
    import torch

    assert torch.cuda.is_available(), "the gpu tests need a CUDA device"
    import knng

    knng.lib()
    return torch, knng


@pytest.mark.parametrize("n,d,leaf,trees,data", [
    (65, 128, 64, 3, "mix"), (511, 128, 64, 2, "mix"), (512, 256, 64, 2, "mix"), (1000, 384, 64, 3, "mix"),
    (5001, 1024, 64, 2, "mix"), (4000, 512, 8, 2, "mix"), (1500, 640, 2, 2, "mix"), (2500, 768, 3, 1, "mix"),
    (9000, 896, 17, 1, "mix"), (700, 128, 64, 1, "same"), (3000, 128, 20, 2, "few"), (64, 128, 64, 2, "mix"),
])
def test_native_forest_equals_restatement(env, n, d, leaf, trees, data):
    torch, knng = env
    if data == "mix":
        x = synth.mixture(n, d, max(3, n // 80), seed=n + leaf)
        codes = np.trunc(x * 127).astype(np.int8)
    elif data == "same":  # no split separates anything: one member per level
        codes = np.full((n, d), 3, np.int8)
    else:  # five distinct rows: ties everywhere
        codes = np.random.default_rng(n).integers(-20, 20, (5, d)).astype(np.int8)[np.arange(n) % 5]
    ref_perm, ref_flags = native_forest(codes, trees, leaf, 1337)
    with knng.Context(leaf_size=leaf, num_trees=trees) as ctx:
        perm, flags = ctx.forest(torch.from_numpy(codes).cuda())
    np.testing.assert_array_equal(perm.cpu().numpy(), ref_perm)
    np.testing.assert_array_equal(flags.cpu().numpy(), ref_flags)
