"""The header reform of batches long enough for the parallel check (2048
packets): sizes around whole 1024-packet tiles, irregular timestamps and runs
of invalid packets at the tiles' edges, two batches in a row.  Packets and
state equal the oracle's, which steps through them one at a time."""
import numpy as np
import pytest

from gpu_util import dev, host
from oracle import sdbe_oracle as O

pytestmark = pytest.mark.gpu

CLK, FRAME = 286_000_000, 262_144


def _batch(n, first_frame, rng):
    """n packets with new-format headers, 256 to a B-frame, across a second boundary."""
    t = 1234 * CLK + CLK - 3 * FRAME + FRAME * (first_frame + np.arange(n) // 256)
    ts = ((t // CLK) << 29) | (t % CLK)
    p = rng.integers(0, 256, (n, 1056), dtype=np.uint8)
    w = p.view("<u4")
    w[:, 0] &= 0x3FFFFFFF
    w[:, 4] = (ts >> 21).astype(np.uint32)
    w[:, 5] = (np.arange(n) % 256 | (rng.integers(0, 8, n) << 8) | ((ts & 0x1FFFFF) << 11)).astype(np.uint32)
    return p


def _shift(p, i, clocks):
    w = p.view("<u4")
    ts = (int(w[i, 4]) << 21) | (int(w[i, 5]) >> 11)
    ts += clocks
    w[i, 4], w[i, 5] = ts >> 21, (int(w[i, 5]) & 0x7FF) | ((ts & 0x1FFFFF) << 11)


def _invalid(p, lo, hi):
    p.view("<u4")[lo:hi, 0] |= np.uint32(1 << 31)


EDITS = {
    "regular": lambda p, n: None,
    "jitter first": lambda p, n: _shift(p, 0, 5),
    "jitter last": lambda p, n: _shift(p, n - 1, 5),
    "jitter at a tile's end": lambda p, n: _shift(p, 1023, 7),
    "jitter at a tile's start": lambda p, n: _shift(p, 1024, 7),
    "first tile invalid": lambda p, n: _invalid(p, 0, 1024),
    "last packets invalid": lambda p, n: _invalid(p, n - 1030, n),
    "a tile before invalid": lambda p, n: _invalid(p, 900, 2047),
    "edge invalid": lambda p, n: _invalid(p, 1020, 1030),
    "all invalid": lambda p, n: _invalid(p, 0, n),
}


@pytest.fixture(scope="module")
def P():
    import __graft_entry__ as g

    g.build()
    from sdbe_gb300 import pac8

    return pac8


@pytest.mark.parametrize("edit", list(EDITS))
@pytest.mark.parametrize("n", [2047, 2048, 2049, 3072, 3073])
def test_reform_equals_oracle(P, n, edit):
    rng = np.random.default_rng(n)
    st, ost = P.new_state(), O.ReformState()
    for k, first in enumerate((0, 2 + n // 256)):
        p = _batch(n, first, rng)
        if k == 0 or edit != "all invalid":
            EDITS[edit](p, n)
        d = dev(p)
        P.beng_reform(st, d, n)
        ref = O.beng_reform_headers(p.copy(), ost)
        got = host(d).reshape(n, 1056)
        bad = np.nonzero((got != ref).any(axis=1))[0]
        assert bad.size == 0, (k, bad[:5])
        assert (st.t0_sec, st.t0_clk, st.tprev_sec, st.tprev_clk) == (*ost.t0, *ost.tprev)
        assert st.bprev == ost.bprev
    if edit in ("regular", "edge invalid"):
        assert st.slow_tiles == 0
