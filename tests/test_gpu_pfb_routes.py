"""The inverse PFB with and without the kept factor: the same results, also in
captured calls, beside larger calls on the same handle, and where memory is
short."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = 32768


@pytest.fixture(scope="module")
def R():
    import __graft_entry__ as g

    g.build()
    from sdbe_gb300 import Resampler

    return Resampler


def _spectra(nb, seed):
    import torch

    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.view_as_complex(torch.randn(nb, L // 2 + 1, 2, device="cuda", generator=gen))


def _inv(r, S, ntap, **kw):
    from sdbe_gb300 import pfb

    return pfb.inverse_pfb(r, S, ntap, **kw)


def _capture(r, S, ntap):
    import torch

    out = torch.zeros((S.shape[0] + ntap - 1, L), device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        _inv(r, S, ntap, out=out, stream=torch.cuda.current_stream().cuda_stream)

    def replay():
        out.zero_()
        g.replay()
        torch.cuda.synchronize()
        return out

    replay.graph = g
    return replay


def _close(a, b):
    """Equal but for the factor's other order of FP64 operations, which moves an
    FP32 result by its last place: 2^-24 of it, and of the whole's RMS for the
    conditioning (up to 3e5 at these sizes, times FP64's 2^-53)."""
    return float((a.double() - b.double()).pow(2).mean().sqrt() / b.double().pow(2).mean().sqrt()) < 2.0 ** -24


def test_captured_call_beside_larger_ones(R):
    """A larger call neither takes a captured call's factor away nor keeps a
    later capture from having one."""
    S, big = _spectra(48, 1), _spectra(4100, 2)
    with R(max_frames=1) as r:
        _inv(r, big, 4)
        ref = _inv(r, S, 4).clone()
        first = _capture(r, S, 4)
        assert bool((first() == ref).all())
        _inv(r, big, 4)
        assert bool((first() == ref).all())
        second = _capture(r, S, 4)
        assert bool((second() == ref).all())
        assert bool((first() == ref).all())


def test_captured_call_that_forms_rows(R):
    """Room from a larger call of other taps, fewer rows formed for these."""
    S = _spectra(100, 3)
    with R(max_frames=1) as fresh:
        ref = _inv(fresh, S, 3).clone()
    with R(max_frames=1) as r:
        _inv(r, S, 4)
        _inv(r, S[:50], 3)
        replay = _capture(r, S, 3)
        for _ in range(2):
            assert bool((replay() == ref).all())
        assert bool((_inv(r, S, 3) == ref).all())
        assert bool((replay() == ref).all())


@pytest.mark.parametrize("ntap", [2, 3, 4, 8])
def test_without_the_kept_factor(R, ntap):
    """A capture on a handle that has seen only a call above 4096 blocks forms
    its factor as it goes."""
    S = _spectra(40, 10 + ntap)
    with R(max_frames=1) as fresh:
        ref = _inv(fresh, S, ntap).clone()
    with R(max_frames=1) as r:
        _inv(r, _spectra(4097, 5), ntap)
        assert _close(_capture(r, S, ntap)(), ref)


@pytest.fixture(scope="module")
def solver(R):
    """A handle whose captured calls of up to 8 spectra form their factor as they go."""
    with R(max_frames=1) as r:
        _inv(r, _spectra(4097, 5), 4)
        yield r


@pytest.mark.parametrize("scale", [0.0, 1e-45, 1e-43, 1e-41, 1e-39, 1e-36, 1.0, 1e30, 2e34, 1e36, "inf row", "nan row"])
def test_values_converted_by_parts(R, solver, scale):
    """Time samples and blocks that are zero, denormal, ordinary, large, beyond
    FP32's range or not finite: the kept factor's integer conversions against
    FP64 instructions.  Tolerance: FP32's last place, and 1e-10 of the RMS for the
    other order of the FP64 operations."""
    import torch

    S = _spectra(8, 77)
    if isinstance(scale, str):
        S[3, 100] = float(scale.split()[0])
    else:
        S = (S.to(torch.complex128) * scale).to(torch.complex64)
    with R(max_frames=1) as r:
        got = _inv(r, S, 4).double()
    ref = _capture(solver, S, 4)().double()
    for test in (torch.isnan, torch.isposinf, torch.isneginf):
        assert torch.equal(test(got), test(ref))
    ok = torch.isfinite(ref)
    if scale == 0.0:
        assert not bool(got.any())
    if not bool(ok.any()):
        return
    a, b = got[ok], ref[ok]
    rms = float(b.pow(2).mean().sqrt()) if float(b.abs().max()) < 1e150 else float(b.abs().max())
    assert bool(((a - b).abs() <= 2.0 ** -23 * b.abs() + 2.0 ** -149 + 1e-10 * rms).all())


@pytest.mark.parametrize("nb", [4096, 4097])
def test_longest_kept_and_shortest_formed_as_it_goes(R, nb):
    """The blocks' forward PFB gives the pseudo time stream again.  A residual
    of FP32 rounding: of the blocks (2^-24, four taps of at most 1 each) and of
    the transform (the stage functions' 4e-7), on the scale of both."""
    import torch

    S = _spectra(nb, nb)
    with R(max_frames=1) as r:
        x = _inv(r, S, 4).double()
    n = torch.arange(4 * L, device="cuda", dtype=torch.float64)
    w = (0.54 - 0.46 * torch.cos(2 * np.pi * n / (4 * L - 1))).view(4, L)
    y = torch.fft.irfft(S.to(torch.complex128), n=L)
    res = sum(w[t] * x[t:t + nb] for t in range(4)) - y
    rms = lambda a: float(a.pow(2).mean().sqrt())
    assert rms(res) <= 4 * 2.0 ** -24 * rms(x) + 4e-7 * rms(y)


def test_short_memory(R):
    """2048 blocks and eight taps need 4.3 GiB as the factor is formed, 0.5 GiB
    more to keep it: with room for the first only, the call succeeds."""
    import torch

    S = _spectra(2048, 6)
    with R(max_frames=1) as fresh:
        ref = _inv(fresh, S, 8).clone()
    out = torch.empty_like(ref)
    with R(max_frames=1) as r:
        _inv(r, S[:1], 8, out=out)  # the library's small buffers and kernels
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        need = 2048 * L * (4 + 64)
        free, _ = torch.cuda.mem_get_info()
        fill = torch.empty(free - need - (256 << 20), dtype=torch.uint8, device="cuda")
        try:
            _inv(r, S, 8, out=out)
        finally:
            del fill
            torch.cuda.empty_cache()
    # the rounding of 2048 blocks' systems: their condition (8e7) times 2^-53, beside FP32's
    d = float((out.double() - ref.double()).pow(2).mean().sqrt() / ref.double().pow(2).mean().sqrt())
    assert d < 8e7 * 2.0 ** -53 * 16 + 2.0 ** -24
