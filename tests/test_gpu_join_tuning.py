"""What the join's autotuner costs a context's first build.

With use_graph = 0 two builds of the same rows launch the same kernels, so the
first build of a (dimension, size) launches more by the tuner's sweeps alone.
"""
import pytest

pytestmark = pytest.mark.gpu


def _tuning_launches(knng, ctx, x):
    counts = []
    for _ in range(2):
        st = knng.Stats()
        ctx.build(x, stats=st)
        counts.append(st.kernel_launches)
    return counts[0] - counts[1]


@pytest.mark.parametrize("k,mult", [(50, 4), (32, 8), (15, 4)])
def test_other_sizes_are_tuned_by_one_launch_per_configuration(k, mult):
    import knng
    import synth

    x = synth.mixture_torch(6001, 384, 60, 3)
    with knng.Context(use_graph=0, k_build=k, rerank_mult=mult) as ctx:
        # five configurations, a launch that fills the candidate cache, five with it
        assert _tuning_launches(knng, ctx, x) <= 11
        assert _tuning_launches(knng, ctx, x) == 0


def test_long_sweeps_are_not_repeated():
    """Beyond 622,592 rows a sweep's launch covers 1/16 of them and takes milliseconds."""
    import knng
    import synth

    x = synth.mixture_torch(640001, 128, 2000, 3)
    with knng.Context(use_graph=0) as ctx:
        assert _tuning_launches(knng, ctx, x) <= 11


def test_tuning_of_a_size_does_not_depend_on_the_sizes_before():
    """82,000 and 123,000 rows of 1024 codes share a power of two, and join_far's line (120 MiB of
    codes) lies between them: each is tuned for itself, whichever is built first."""
    import knng
    import synth

    seen = []
    for order in ((82000, 123000), (123000, 82000)):
        with knng.Context(use_graph=0) as ctx:
            seen.append({n: _tuning_launches(knng, ctx, synth.mixture_torch(n, 1024, n // 300, 4)) for n in order})
    assert seen[0] == seen[1]
