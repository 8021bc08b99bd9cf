"""The join's duplicate tables when their tags are worn out.

A CTA clears its tables once per about 300,000 rows.  The bounds-checked
library starts with a few dozen tags more than a row may use, so its CTAs
clear them every dozen rows or so; its iterations must equal the default
library's, for the default form, the form for codes beyond L2 and the general
form.  The checked library runs in a child process.
"""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

import synth
from test_gpu_checked import PKG, ROOT, checked_lib  # noqa: F401  (fixture)
from test_gpu_join_forms import LAUNCH_JOIN

pytestmark = pytest.mark.gpu
N, D = 30011, 128  # about 50 rows per CTA
SIZES = [(50, 8), (50, 5), (64, 8), (20, 3)]


def iterations():
    """Two iterations of every form: {name: array}."""
    import torch

    import knng

    codes, sk = knng.quantize(torch.from_numpy(synth.mixture(N, D, 600, seed=8)).cuda())
    out = {}
    for k, mult in SIZES:
        with knng.Context(k_build=k, rerank_mult=mult) as ctx:
            perm, lf = ctx.forest(codes)
            ids, sc = ctx.init_graph(codes, perm, lf)
            start = (ids, sc)
            for it in range(2):
                ids, sc, up = ctx.join_iter(codes, sk, ids, sc)
                out[f"{k}_{mult}_{it}"] = np.stack([ids.cpu().numpy(), sc.cpu().numpy()])
                assert up > 0
        if (k, mult) == (50, 8):
            far = start
            launch = C.CDLL(knng.LIB_PATH)[LAUNCH_JOIN]
            launch.restype = C.c_int
            sms = torch.cuda.get_device_properties(0).multi_processor_count
            ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
            for it in range(2):
                to = (torch.empty_like(far[0]), torch.empty_like(far[1]))
                counters = torch.zeros(8, dtype=torch.int64, device="cuda")
                torch.cuda.synchronize()
                assert launch(ptr(codes), ptr(sk), C.c_int64(N), C.c_int(D), C.c_int(k), C.c_int(k * mult), ptr(far[0]),
                              ptr(far[1]), ptr(to[0]), ptr(to[1]), None, ptr(counters), C.c_int(sms), None, None, None,
                              C.c_int(4), C.c_int(4), C.c_int(0), C.c_bool(True)) == 0
                torch.cuda.synchronize()
                far = to
                out[f"far_{it}"] = np.stack([far[0].cpu().numpy(), far[1].cpu().numpy()])
    return out


def test_worn_tags_change_nothing(checked_lib, tmp_path):  # noqa: F811
    ref = iterations()
    assert all(np.array_equal(ref[f"far_{it}"], ref[f"50_8_{it}"]) for it in range(2))
    npz = str(tmp_path / "checked.npz")
    code = (f"import sys; sys.path[:0] = [{PKG!r}, {os.path.join(ROOT, 'oracle')!r}, {os.path.join(ROOT, 'tests')!r}]\n"
            "import numpy as np, knng, test_gpu_join_tags as t\n"
            "assert knng.LIB_PATH.endswith('libknng_checked.so')\n"
            f"np.savez({npz!r}, **t.iterations())\n")
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, KNNG_LIBRARY=checked_lib), cwd=ROOT,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    got = np.load(npz)
    for name, a in ref.items():
        np.testing.assert_array_equal(got[name], a, err_msg=name)
