"""The two-channel residual as matrix products (two_channel_mm.cu) against the oracle, term by
term, at the sizes where its tiles and groups can go wrong: one occupied orbital (no pair of
distinct orbitals), a basis below one 64-wide tile, one that ends inside a tile, odd orbital
counts; with equal and with different direct and exchange flags; and with values at amplitudes
that have no virtual partner, which every term ignores.  Tolerance as in
test_gpu_two_channel.py: 1e-12 of the largest element."""
import numpy as np
import pytest

from oracle.oracle import Oracle, parse_input_text
from test_gpu_two_channel import KEYS, MIXED, _screening
from uegccd_b200 import Context
from uegccd_b200 import _capi as capi

pytestmark = pytest.mark.gpu

SAME = dict(ring=1, xring=1, ladder=1, mosaic=1, driver_direct=1, driver_exchange=1, energy=1)


@pytest.mark.parametrize("flags", [None, SAME, MIXED], ids=["plain", "same flags", "mixed flags"])
@pytest.mark.parametrize("nel,cut", [(2, 3), (14, 2), (14, 5), (30, 6), (38, 8)])
def test_every_term_matches_oracle(nel, cut, flags):
    v = parse_input_text("")
    v.update({"# Electrons": str(nel), "Momentum Cutoff": str(cut), "rSMin": "2.0", "rSMax": "2.0",
              "Safe ERI": "T" if flags else "F"})
    for k, name in zip(KEYS, capi.RANGE_TERMS):
        v[k] = str((flags or {}).get(name, 0))
    o = Oracle(v)
    o.change_twist((0.11, -0.23, 0.31))
    sc = o.scalars()
    ctx = Context(o.nocc, sc["L"], sc["madelung"], o.eigen(), o.nvec())
    if flags:
        ctx.set_eri(flags, safe_eri=True, screening=_screening(2 * o.nocc, sc["L"]))
    rng = np.random.default_rng(nel + cut)
    _, _, tb, tc, _ = o.mp2()
    tb = tb + 1e-3 * rng.standard_normal(tb.shape)
    tc = tc + 1e-3 * rng.standard_normal(tc.shape)
    for mask in (1, 2, 4, 8, 16, 31):
        ga, gb = o.ccd_g2(tb, tc, mask)
        ha, hb = ctx.ccd_g2_2ch(tb, tc, mask)
        scale = max(np.abs(ga).max(), np.abs(gb).max())
        assert np.abs(ha - ga).max() <= 1e-12 * scale, (mask, "abab")
        assert np.abs(hb - gb).max() <= 1e-12 * scale, (mask, "abba")
