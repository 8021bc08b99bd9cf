"""The join's forms for codes beyond L2, at sizes where the oracle is quick.

A build takes one of them (four CTAs per SM, 4 or 8 sketches in flight) where
the tuner or the size says so, and no parameter forces them; they are launched
here through the library's own launcher.  Each must equal the oracle's
double-buffered, stable-tie iteration (src/main.cpp:320-440) bit for bit.
"""
import ctypes as C

import numpy as np
import pytest

import oracle
import synth

pytestmark = pytest.mark.gpu
LAUNCH_JOIN = ("_ZN4knng11launch_joinEPKaPKmliiiPKiS5_PiS6_S5_PyiP11CUstream_stPKNS_8JobTableE"
               "PKNS_7JoinCtlEiiib")


@pytest.mark.parametrize("cblock", [4, 8])
@pytest.mark.parametrize("n,d", [(4001, 1024), (3000, 384), (2503, 128)])
def test_far_form_iterations_bit_exact(cblock, n, d):
    import torch

    import knng

    knng.lib()
    launch = C.CDLL(knng.LIB_PATH)[LAUNCH_JOIN]
    launch.restype = C.c_int
    codes_h, sk_h = oracle.quantize(synth.mixture(n, d, n // 20, seed=n))
    prm = oracle.params(threads=1, tie_mode=oracle.TIE_STABLE, jacobi=1)
    perm, lf, _ = oracle.forest(codes_h, prm)
    ids_ref, sc_ref = oracle.init_graph(codes_h, perm, lf, prm)
    codes, sk = torch.from_numpy(codes_h).cuda(), torch.from_numpy(sk_h.view(np.int64)).cuda()
    ids, sc = torch.from_numpy(ids_ref.copy()).cuda(), torch.from_numpy(sc_ref.copy()).cuda()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    for it in range(3):
        up_ref = oracle.join_iter(codes_h, sk_h, ids_ref, sc_ref, prm)
        out, out_sc = torch.empty_like(ids), torch.empty_like(sc)
        counters = torch.zeros(8, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        err = launch(ptr(codes), ptr(sk), C.c_int64(n), C.c_int(d), C.c_int(50), C.c_int(400), ptr(ids), ptr(sc),
                     ptr(out), ptr(out_sc), None, ptr(counters), C.c_int(sms), None, None, None, C.c_int(4),
                     C.c_int(cblock), C.c_int(0), C.c_bool(True))
        assert err == 0
        torch.cuda.synchronize()
        assert int(counters[0]) == up_ref, f"iteration {it}"
        np.testing.assert_array_equal(out_sc.cpu().numpy(), sc_ref)
        np.testing.assert_array_equal(out.cpu().numpy(), ids_ref)
        ids, sc = out, out_sc
