"""The join's form for codes beyond L2 against the general form.

Lists that start on an 8-byte boundary take the form for the default K and R;
from 120 MiB of codes on that is the one with less shared memory per CTA.  The
same lists 4 bytes further on take the general form, which
test_gpu_join_table.py compares with the oracle.  Both must agree bit for bit,
also on starting lists in ascending order, whose survivors are inserted one by
one, and a build with the candidate cache must equal one without it.
"""
import pytest

pytestmark = pytest.mark.gpu
SHAPES = [(123000, 1024), (330000, 384), (990000, 128)]


@pytest.mark.parametrize("n,d", SHAPES)
@pytest.mark.parametrize("ascending", [False, True])
def test_far_form_equals_general_form(n, d, ascending):
    import torch

    import knng
    import synth

    assert n * d >= 120 << 20
    x = synth.mixture_torch(n, d, n // 300, 5)
    codes, sk = knng.quantize(x)
    del x

    def at_offset(a, offset):
        buf = torch.empty(a.numel() + offset, dtype=torch.int32, device="cuda")
        out = buf[offset:].view(a.shape)
        out.copy_(a)
        return out

    with knng.Context() as ctx:
        perm, lf = ctx.forest(codes)
        ids, sc = ctx.init_graph(codes, perm, lf)
        if ascending:
            ids, sc = ids.flip(1).contiguous(), sc.flip(1).contiguous()
        far, gen = (ids, sc), (at_offset(ids, 1), at_offset(sc, 1))
        for it in range(2):
            fi, fs, fu = ctx.join_iter(codes, sk, *far, torch.empty_like(ids), torch.empty_like(sc))
            gi, gs, gu = ctx.join_iter(codes, sk, *gen, at_offset(ids, 1), at_offset(sc, 1))
            assert fi.data_ptr() % 8 == 0 and gi.data_ptr() % 8 == 4
            assert fu == gu and fu > 0, f"iteration {it}"
            assert torch.equal(fi, gi) and torch.equal(fs, gs)
            far, gen = (fi, fs), (gi, gs)


@pytest.mark.parametrize("n,d", SHAPES[:2])
def test_far_build_with_cache_equals_build_without(n, d):
    import torch

    import knng
    import synth

    x = synth.mixture_torch(n, d, n // 300, 6)
    got = []
    for cache in (0, 1):
        with knng.Context(join_cache=cache) as ctx:
            st = knng.Stats()
            k, dd, _ = ctx.build(x, stats=st)
        got.append((k, dd, list(st.updates[: st.iterations])))
    assert torch.equal(torch.as_tensor(got[0][0]), torch.as_tensor(got[1][0]))
    assert torch.equal(torch.as_tensor(got[0][1]), torch.as_tensor(got[1][1]))
    assert got[0][2] == got[1][2]
