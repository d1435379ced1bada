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
def test_calls_that_wait_report_it(N, stream, stage):
    """A call that synchronizes reports its own time-out, as does sdbe_sync."""
    import torch

    from sdbe_gb300 import Resampler

    p, b0, _ = stream
    for host in (True, False):
        with Resampler(trim_mhz=150, max_frames=2) as rs:
            N.check(N.lib().sdbe_test_fft_timeout(rs.handle, stage), rs.handle)
            if host:
                _timed_out(N, lambda: rs.process(p[:4096], 2, b0))
            else:
                out = torch.empty(rs.output_bytes(2), dtype=torch.uint8, device="cuda")
                rs.process(torch.from_numpy(p[:4096]).cuda(), 2, b0, out=out, want_result=False)
                _timed_out(N, rs.sync)


@pytest.mark.parametrize("stage,name", [(1, "sdbe_swarm_c2r"), (2, "sdbe_resample_chunks")])
def test_stage_functions_report_it(N, stage, name):
    import torch

    from sdbe_gb300 import Resampler

    n = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 1  # fewer chunks run without waits
    a, b = (torch.zeros(n * 36608, device="cuda") for _ in range(2))
    with Resampler(max_frames=2) as rs:
        N.check(N.lib().sdbe_test_fft_timeout(rs.handle, stage), rs.handle)
        fn = getattr(N.lib(), name)
        assert fn(rs.handle, a.data_ptr(), n, b.data_ptr(), None) == N.OK
        _timed_out(N, rs.sync)
        assert fn(rs.handle, a.data_ptr(), n, b.data_ptr(), None) == N.ERR_CUDA


@pytest.mark.parametrize("stage", [1, 2])
def test_ingest_reports_it(N, stage):
    from sdbe_gb300 import Resampler, synth

    spec = synth.config1()
    spec.n_frames = 4
    p = synth.generate(spec)
    with Resampler(max_frames=143) as rs:
        rs.ingest(p)
        N.check(N.lib().sdbe_test_fft_timeout(rs.handle, stage), rs.handle)
        _timed_out(N, rs.ingest_flush)


@pytest.mark.parametrize("waits", [False, True])
@pytest.mark.parametrize("precision", ["FP32-1", "FP32-2", "TC16_FAST"])
def test_every_handle_of_a_shared_launch_reports_it(N, stream, precision, waits):
    """The first handle's launches time out; one handle has no batch in them."""
    import torch

    from sdbe_gb300 import Resampler
    from sdbe_gb300.resampler import process_multi

    p, b0, _ = stream
    name, _, stage = precision.partition("-")
    rs = [Resampler(max_frames=2, precision=getattr(N, "PRECISION_" + name)) for _ in range(4)]
    if stage:
        N.check(N.lib().sdbe_test_fft_timeout(rs[0].handle, int(stage)), rs[0].handle)
    else:
        N.check(N.lib().sdbe_test_tc_timeout(rs[0].handle, 2_000_000), rs[0].handle)
    d = torch.from_numpy(p[:4096]).cuda()
    outs = [torch.empty(r.output_bytes(2), dtype=torch.uint8, device="cuda") for r in rs]
    torch.cuda.synchronize()
    items = [(d, 2 if i != 1 else 1, b0, outs[i]) for i in range(3)]  # one frame: no batch
    if waits:
        _timed_out(N, lambda: process_multi(rs[:3], items, want_results=True))
        for i in (0, 2):
            _timed_out(N, lambda: rs[i].process(d, 1, b0, out=outs[i]))
    else:
        process_multi(rs[:3], items)
        for i in (0, 2):
            _timed_out(N, rs[i].sync)
    for i in (1, 3):
        rs[i].sync()
    assert rs[1].get_state().carry_snapshots == 128
    for r in rs:
        r.close()


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
