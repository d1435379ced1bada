"""The inverse PFB's kept factor: calls that form it, reuse it, extend it or
replace it (fewer and more blocks, other taps, fewer blocks than taps) against
the FP64 oracle, and reuse against a fresh handle bit for bit.  Tolerance as in
test_gpu_pfb: the FP32 input's error times the conditioning."""
import numpy as np
import pytest

from oracle import sdbe_oracle as O

pytestmark = pytest.mark.gpu

L = 32768
TOL = 1e-4


def _spectra(ntap, nb, seed):
    x = np.random.default_rng(seed).standard_normal((nb + ntap - 1) * L)
    return O.forward_pfb(x, L, ntap).astype(np.complex64)


def test_factor_kept_extended_and_replaced():
    import __graft_entry__ as g

    g.build()
    from sdbe_gb300 import Resampler, pfb

    with Resampler(max_frames=1) as r:
        for k, (ntap, nb) in enumerate([(4, 3), (4, 3), (4, 9), (4, 2), (8, 2), (8, 5), (3, 1), (4, 9)]):
            S = _spectra(ntap, nb, 100 + k)
            got = pfb.inverse_pfb(r, S, ntap=ntap).cpu().numpy()
            with Resampler(max_frames=1) as fresh:
                assert np.array_equal(got, pfb.inverse_pfb(fresh, S, ntap=ntap).cpu().numpy()), (ntap, nb)
            ref = O.inverse_pfb(S.astype(np.complex128), ntap)
            err = np.sqrt(np.mean((got - ref) ** 2) / np.mean(ref ** 2))
            assert err < TOL, (ntap, nb, err)


def test_zeros_denormals_and_large_values():
    """Spectra whose time samples are zero, tiny or large: the conversion to FP64 by parts."""
    import __graft_entry__ as g

    g.build()
    from sdbe_gb300 import Resampler, pfb

    S = _spectra(4, 6, 7)
    S[1] = 0
    S[2] *= np.float32(1e-38)
    S[3] *= np.float32(1e30)
    with Resampler(max_frames=1) as r:
        got = pfb.inverse_pfb(r, S, ntap=4).cpu().numpy()
    ref = O.inverse_pfb(S.astype(np.complex128), 4)
    err = np.sqrt(np.mean((got - ref) ** 2) / np.mean(ref ** 2))
    assert err < TOL, err


@pytest.mark.parametrize("ntap,nb", [(n, b) for n in (2, 4, 8) for b in (1, 3, 4, 5, 8)])
@pytest.mark.parametrize("scale", [1.0, 1e-41])
def test_rows_in_flight_and_small_results(ntap, nb, scale):
    """Fewer, as many and more rows than are in flight at once; results among
    FP32's normal numbers, and around the smallest of them (rounded by parts).
    Tolerance as above, plus FP32's spacing of 2^-149 there."""
    import __graft_entry__ as g

    g.build()
    from sdbe_gb300 import Resampler, pfb

    S = (_spectra(ntap, nb, 40 + ntap) * scale).astype(np.complex64)
    with Resampler(max_frames=1) as r:
        got = pfb.inverse_pfb(r, S, ntap=ntap).cpu().numpy().astype(np.float64)
    ref = O.inverse_pfb(S.astype(np.complex128), ntap)
    assert np.sqrt(np.mean((got - ref) ** 2)) < TOL * np.sqrt(np.mean(ref ** 2)) + 2.0 ** -149
