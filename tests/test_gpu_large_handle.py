"""Handles whose two phased sums lie more than a 2D copy's largest pitch
(2 GiB) apart: the leftover snapshots are carried as on a small handle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def S():
    import __graft_entry__ as g

    g.build()
    from sdbe_gb300 import synth

    return synth


def _two_calls(p, b0, max_frames):
    from sdbe_gb300 import Resampler

    with Resampler(trim_mhz=150, max_frames=max_frames) as rs:
        out = [rs.process(p[k * 4096:(k + 1) * 4096], 2, b0 + 2 * k) for k in range(2)]
        return np.concatenate([o for o, _ in out], axis=1), [r.carry_snapshots for _, r in out], rs.thresholds


@pytest.mark.parametrize("max_frames", [2046, 2047])
def test_carry_of_a_large_handle(S, max_frames):
    """(128 max_frames + 143) * 8192 bytes: just below and just above 2^31 - 1."""
    spec = S.config1()
    spec.n_frames = 4
    p = S.generate(spec)
    ref = _two_calls(p, spec.b_start, 4)
    got = _two_calls(p, spec.b_start, max_frames)
    assert ref[1] == [113, 83]
    assert got[1:] == ref[1:]
    assert np.array_equal(got[0], ref[0])
