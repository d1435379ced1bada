"""Bounded barrier waits of the FP32 kernels (failure detection without a GPU
fault): ``sdbe_test_fft_timeout`` has a stage expect one barrier arrival that
never comes.  Its waits run out after one second, the kernel records that,
lets its copies land, frees its tensor memory and returns; the handle's later
calls fail, and a fresh handle works on as before."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

@pytest.fixture(scope="module")
def N():
    import __graft_entry__ as g

    g.build()
    from sdbe_gb300 import _native

    return _native


@pytest.fixture(scope="module")
def stream(N):
    from sdbe_gb300 import Resampler, synth

    spec = synth.config1()
    spec.n_frames = 8
    p = synth.generate(spec)
    with Resampler(trim_mhz=150, max_frames=8) as rs:
        out, _ = rs.process(p, 8, spec.b_start)
    return p, spec.b_start, out


def _timed_out(N, call):
    with pytest.raises(N.SdbeError) as ei:
        call()
    assert ei.value.code == N.ERR_CUDA and "timed out" in str(ei.value), ei.value


def test_hook_refuses_bad_arguments(N):
    from sdbe_gb300 import Resampler

    lib = N.lib()
    assert lib.sdbe_test_fft_timeout(None, 1) == N.ERR_ARG
    with Resampler(max_frames=2) as rs:
        for stage in (0, 3):
            assert lib.sdbe_test_fft_timeout(rs.handle, stage) == N.ERR_ARG


@pytest.mark.parametrize("stage", [1, 2])
def test_wait_that_runs_out(N, stream, stage):
    """Launches of several items per CTA and of one; then a fresh handle."""
    from sdbe_gb300 import Resampler

    p, b0, ref = stream
    with Resampler(trim_mhz=150, max_frames=8) as rs:
        N.check(N.lib().sdbe_test_fft_timeout(rs.handle, stage), rs.handle)
        t0 = time.perf_counter()
        try:
            rs.process(p, 8, b0)
        except N.SdbeError as e:
            assert e.code == N.ERR_CUDA, e
        elapsed = time.perf_counter() - t0
        _timed_out(N, lambda: rs.process(p, 8, b0))
    assert elapsed < 4.0, elapsed  # two launches, one wait each
    with Resampler(trim_mhz=150, max_frames=8) as rs:
        out, _ = rs.process(p, 8, b0)
    assert np.array_equal(out, ref)
