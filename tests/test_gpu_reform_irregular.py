"""The header reform of irregular batches, walked tile by tile and after the
parallel check (from 4096 packets on): clocks outside the second, seconds
apart, values at the comparison's tolerance, jumps beyond the cap and back,
random timestamps.  Packets and state equal the oracle's, which steps through
them one at a time."""
import numpy as np
import pytest

from gpu_util import dev, host
from oracle import sdbe_oracle as O

pytestmark = pytest.mark.gpu

CLK, FRAME, TOL = 286_000_000, 262_144, 1024


def _packets(sec, clk, rng):
    n = sec.size
    p = rng.integers(0, 256, (n, 1056), dtype=np.uint8)
    ts = (sec.astype(np.int64) << 29) | clk
    w = p.view("<u4")
    w[:, 0] = (w[:, 0] & 0x3FFFFFFF) | (np.uint32(1 << 31) * (rng.random(n) < 0.05)).astype(np.uint32)
    w[:, 4] = (ts >> 21).astype(np.uint32)
    w[:, 5] = (np.arange(n) % 256 | (rng.integers(0, 8, n) << 8) | ((ts & 0x1FFFFF) << 11)).astype(np.uint32)
    return p


def _times(kind, n, rng):
    t = 1234 * CLK + CLK - 9 * FRAME + FRAME * (np.arange(n) // 256)
    if kind == "edges":
        edge = np.array([CLK - TOL, CLK - TOL + 1, CLK - TOL - 1, CLK, CLK + 5, 2**29 - 1, 0, TOL - 1, TOL, TOL + 1,
                         FRAME, CLK - FRAME])
        return 500 + rng.integers(0, 3, n), edge[rng.integers(0, edge.size, n)]
    if kind == "random":
        return 1234 + rng.integers(0, 2, n), rng.integers(0, 2**29, n)
    if kind == "jumps":
        t = t + FRAME * rng.choice([0, 0, 0, 0, 0, 0, 0, 3, 999, 1000, 1001, 1002, 1003, 1200, -1000, -1001, -1003], n)
    if kind == "jitter":
        t = t + rng.integers(-1500, 1501, n)
    if kind == "one far":
        t[n // 2] += 40 * CLK
    if kind == "last far":
        t[[1023, n - 1]] += 40 * CLK
    return t // CLK, t % CLK


@pytest.mark.parametrize("kind,n", [(k, n) for k in ("edges", "random", "jumps") for n in (1, 700, 1500)]
                         + [("edges", 4096)]
                         + [(k, n) for k in ("regular", "jitter", "one far", "last far")
                            for n in (1024, 4095, 4096, 4097, 5121)])
def test_irregular_batches_equal_oracle(kind, n):
    import __graft_entry__ as g

    g.build()
    from sdbe_gb300 import pac8

    rng = np.random.default_rng(n)
    st, ost = pac8.new_state(), O.ReformState()
    for _ in range(2):
        p = _packets(*_times(kind, n, rng), rng)
        d = dev(p)
        pac8.beng_reform(st, d, n)
        ref = O.beng_reform_headers(p.copy(), ost)
        bad = np.nonzero((host(d).reshape(n, 1056) != ref).any(axis=1))[0]
        assert bad.size == 0, bad[:5]
        assert (st.t0_sec, st.t0_clk, st.tprev_sec, st.tprev_clk) == (*ost.t0, *ost.tprev)
        assert st.bprev == ost.bprev
