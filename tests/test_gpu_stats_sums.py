"""Sums of the summary statistics: no further from exact sums than FP64 sums
of the same samples, split over the threads in the same way."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = 304 * 256  # of the kernel; thread t takes samples t, t + THREADS, ...


@pytest.fixture(scope="module")
def N():
    import __graft_entry__ as g

    g.build()
    from sdbe_gb300 import _native

    return _native


def _stats(N, t):
    out = (C.c_double * 2)()
    N.check(N.lib().sdbe_summary_stats(t.data_ptr(), t.numel(), out, C.c_void_p(1)))
    return out[0], out[1]


@pytest.mark.parametrize("per_thread", [14, 256])
def test_wide_range_of_magnitudes(N, per_thread):
    """Log-normal samples.  Tolerance: the FP64 sums' own error, and 2^-50 for
    the adding up of 304 block sums and the roundings of the result."""
    import torch

    x = np.random.default_rng(per_thread).lognormal(0, 6, (per_thread, THREADS)).astype(np.float32)
    x[0, 0] = 0  # the shift
    s = np.zeros(THREADS)
    for row in x:
        s += row
    exact = math.fsum(x.astype(np.float64).ravel())
    tol = abs(math.fsum(s) - exact) / exact + 2.0 ** -50
    mean, _ = _stats(N, torch.from_numpy(x).cuda())
    assert abs(mean * x.size - exact) <= tol * exact


@pytest.mark.parametrize("n", [1 << 20, 1 << 30])
def test_long_constant_after_another_first_sample(N, n):
    """x[0] = 0 and n - 1 samples of float32(0.1): closed forms.  FP64 sums of a
    thread's N samples are off by N 2^-53 at most."""
    import torch

    t = torch.full((n,), 0.1, device="cuda")
    t[0] = 0
    mean, std = _stats(N, t)
    a = float(np.float32(0.1))
    tol = -(-n // THREADS) * 2.0 ** -53 + 2.0 ** -50
    assert abs(mean / (a * (n - 1) / n) - 1) <= tol
    # M2 = a^2 (n - 1) / n: the difference of two sums n times as large
    assert abs(std / (a / math.sqrt(n)) - 1) <= 2 * n * tol


@pytest.mark.parametrize("kind", ["large", "small", "mixed", "inf", "nan"])
@pytest.mark.parametrize("n", [2, 255, 257, 100_000])
def test_samples_beyond_fp32_squares(N, n, kind):
    """Differences of 1e12 and above or below 1e-10 (FP64 sums), beside ordinary
    ones in the same block; infinities and NaN as FP64 arithmetic has them.
    Tolerance: FP64's, N 2^-53 a sum, the variance's cancellation included."""
    import torch

    rng = np.random.default_rng(n)
    x = rng.standard_normal(n).astype(np.float32)
    x[0] = 0
    if kind == "large":
        x[1:] *= np.float32(1e30)
    elif kind == "small":
        x[1:] *= np.float32(1e-30)
    elif kind == "mixed":
        x[1::2] *= np.float32(1e13)
        x[2::3] *= np.float32(1e-13)
    else:
        x[n // 2] = np.float32(kind)
    mean, std = _stats(N, torch.from_numpy(x).cuda())
    if kind in ("inf", "nan"):
        assert (math.isnan(mean) if kind == "nan" else mean == math.inf) and math.isnan(std)
        return
    d = x.astype(np.float64)
    s1, s2, a1 = math.fsum(d), math.fsum(d * d), math.fsum(np.abs(d))
    tol = n * 2.0 ** -53
    assert abs(mean - s1 / n) <= tol * a1 / n
    m2 = s2 - s1 * s1 / n
    assert abs(std * std * (n - 1) - m2) <= 8 * tol * (s2 + a1 * a1 / n)
