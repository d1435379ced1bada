"""The pipelined FP32 FFT kernels where their pipelines begin, wrap and end:
item counts around one, two and three rounds of the grid (one CTA per SM), each
transform against the same transform alone (bit for bit) and against FP64; and
the 2-bit packing in the stage-BC epilogue against sdbe_quantize2bit, which
compares and selects, at thresholds and offsets where sign tricks can go wrong.
"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

NA, NB = 32768, 36608
LEGACY = C.c_void_p(1)


@pytest.fixture(scope="module")
def env():
    import __graft_entry__ as g

    g.build()
    import torch

    from sdbe_gb300 import Resampler, _native as N

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return torch, N, Resampler, sms


def _counts(sms):
    return {"one": 1, "two": 2, "round": sms, "round+1": sms + 1, "two rounds": 2 * sms, "three rounds+1": 3 * sms + 1}


CASES = ["one", "two", "round", "round+1", "two rounds", "three rounds+1"]


def _c2r(torch, N, rs, spec):
    out = torch.full((spec.shape[0], NA), float("nan"), device="cuda")
    N.check(N.lib().sdbe_swarm_c2r(rs.handle, spec.data_ptr(), spec.shape[0], out.data_ptr(), LEGACY))
    return out


def _resample(torch, N, rs, x):
    out = torch.full((x.shape[0], NA), float("nan"), device="cuda")
    N.check(N.lib().sdbe_resample_chunks(rs.handle, x.data_ptr(), x.shape[0], out.data_ptr(), LEGACY))
    return out


def _rel(got, ref):
    return float((got.double() - ref).norm() / ref.norm())


@pytest.mark.parametrize("case", CASES)
def test_stage_a_item_counts(env, case):
    torch, N, Resampler, sms = env
    n = _counts(sms)[case]
    g = torch.Generator(device="cuda").manual_seed(n)
    spec = torch.randint(-2**31, 2**31 - 1, (n, 2048), device="cuda", generator=g, dtype=torch.int32)
    with Resampler(max_frames=2) as rs:
        out = _c2r(torch, N, rs, spec)
        for i in {0, n // 2, n - 1}:
            assert torch.equal(out[i], _c2r(torch, N, rs, spec[i:i + 1].contiguous())[0]), i
    i = n - 1
    nib = (spec[i][:, None] >> (4 * torch.arange(8, device="cuda"))) & 15
    z = torch.zeros(16385, dtype=torch.complex128, device="cuda")
    z[:-1] = torch.complex((nib >> 2).double() - 2, (nib & 3).double() - 2).reshape(-1)
    assert _rel(out[i], torch.fft.irfft(z, n=NA, norm="forward")) < 2e-6  # the bar of each FFT stage


@pytest.mark.parametrize("trim", [0, 150, 240])
@pytest.mark.parametrize("case", CASES)
def test_stage_bc_item_counts(env, case, trim):
    torch, N, Resampler, sms = env
    n = _counts(sms)[case]
    g = torch.Generator(device="cuda").manual_seed(n + trim)
    x = torch.randn((n, NB), device="cuda", generator=g)
    with Resampler(trim_mhz=trim, max_frames=2) as rs:
        out = _resample(torch, N, rs, x)
        for i in {0, n // 2, n - 1}:
            assert torch.equal(out[i], _resample(torch, N, rs, x[i:i + 1].contiguous())[0]), i
        s = rs.skip_chan
    z = torch.fft.rfft(x[n - 1].double())
    assert _rel(out[n - 1], torch.fft.irfft(z[s:s + 16385], n=NA, norm="forward")) < 2e-6


@pytest.mark.parametrize("precision", ["fp32", "tc16_fast"])
@pytest.mark.parametrize("th,off", [(6e5, 0.0), (6e5, -2e5), (1.0, 0.0), (1e-38, 3e-39), (float("inf"), 0.0),
                                    (float("nan"), 1e5), (6e5, float("inf")), (6e5, float("nan")), (-1.0, 0.0),
                                    (float("nan"), float("-inf")), (float("inf"), float("inf"))])
def test_packing_equals_quantize2bit(env, th, off, precision):
    """sdbe_process with fixed thresholds against the stage functions and sdbe_quantize2bit."""
    torch, N, Resampler, sms = env
    g = torch.Generator(device="cuda").manual_seed(7)
    frames, b0 = 2, 1000
    pk = torch.randint(0, 256, (frames * 2048, 1056), device="cuda", generator=g, dtype=torch.uint8)
    w = pk.view(torch.int32).view(frames, 256, 8, 264)
    w[..., :8] = 0
    b = b0 + torch.arange(frames, device="cuda").int()
    w[..., 4] = (b >> 8)[:, None, None]
    cf = torch.arange(256, device="cuda").int()[:, None] | (torch.arange(8, device="cuda").int()[None] << 16)
    w[..., 5] = cf[None] | ((b & 255) << 24)[:, None, None]
    prec = {"fp32": N.PRECISION_FP32, "tc16_fast": N.PRECISION_TC16_FAST}[precision]
    with Resampler(max_frames=frames, threshold_mode=N.THRESH_FIXED, precision=prec) as rs:
        rs.set_thresholds((th, th), (off, off))
        out, _ = rs.process(pk, frames, b0, out=torch.zeros(2 * 128 * 8192, dtype=torch.uint8, device="cuda"))
        spec = torch.zeros((2, frames * 128, 2048), dtype=torch.int32, device="cuda")
        ints = torch.zeros(frames * 65 + 1, dtype=torch.int32, device="cuda")
        N.check(N.lib().sdbe_unpack(pk.data_ptr(), pk.shape[0], b0, frames, 0, spec.data_ptr(), spec.stride(0), 0,
                                    ints.data_ptr(), ints.data_ptr() + frames * 256, ints.data_ptr() + frames * 260,
                                    LEGACY))
        words = []
        for pol in range(2):
            x = _c2r(torch, N, rs, spec[pol][:143].contiguous()).view(-1, NB)
            y = _resample(torch, N, rs, x)
            o = torch.zeros(128 * 2048, dtype=torch.int32, device="cuda")
            N.check(N.lib().sdbe_quantize2bit(y.data_ptr(), o.data_ptr(), y.numel(), th, off, LEGACY))
            words.append(o)
    assert torch.equal(out.view(torch.int32), torch.cat(words))
