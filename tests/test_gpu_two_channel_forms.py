"""Which form the two-channel residual takes -- matrix products where no integral in use is excluded,
else the loops -- and its values with equal and with different direct and exchange integrals.

An integral is excluded where it is negative under Safe ERI.  Flags 1 (short range) and 3 (none) never
give one; flag 0 gives -Madelung at |q|^2 = 0, negative with a negative MadelungFactor.  Tolerance as
in test_gpu_two_channel.py."""
import numpy as np
import pytest

from oracle.oracle import Oracle, parse_input_text
from profiled import profiled
from test_gpu_two_channel import KEYS, MIXED, _screening
from uegccd_b200 import Context
from uegccd_b200 import _capi as capi

pytestmark = pytest.mark.gpu

ONE = {name: 1 for name in ("ring", "xring", "ladder", "mosaic", "driver_direct", "driver_exchange", "energy")}
FORMS = {   # flags, MadelungFactor, whether the products serve them
    "plain": (None, 1, True),
    "short range": (ONE, 1, True),
    "exchange ladders none": (dict(ONE, exchange_ladders=3), 1, True),
    "direct ladders none": (dict(ONE, direct_ladders=3), 1, True),
    "linear ladders none, exchange rings none": (dict(ONE, lin_ladders=3, exchange_rings=3, quad_rings=3), 1, True),
    "flags 0 to 2": (MIXED, 1, True),
    "short range, Madelung excluded": (ONE, -1, True),
    "one term with an excluded integral": (dict(ONE, mosaic=0), -1, False),
    "flags 0 to 2, excluded integrals": (MIXED, -1, False),
}


def _setup(nel, cut, flags, factor=1):
    v = parse_input_text("")
    v.update({"MadelungFactor": str(factor), "# Electrons": str(nel), "Momentum Cutoff": str(cut), "rSMin": "2.0", "rSMax": "2.0",
              "Safe ERI": "T" if flags else "F"})
    for k, name in zip(KEYS, capi.RANGE_TERMS):
        v[k] = str((flags or {}).get(name, 0))
    o = Oracle(v)
    o.change_twist((0.11, -0.23, 0.31))
    return o


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("nel,cut", [(14, 5), (38, 8)])
def test_terms_and_form(nel, cut, form):
    flags, factor, products = FORMS[form]
    o = _setup(nel, cut, flags, factor)
    sc = o.scalars()
    ctx = Context(o.nocc, sc["L"], sc["madelung"], o.eigen(), o.nvec())
    if flags:
        ctx.set_eri(flags, safe_eri=True, screening=_screening(2 * o.nocc, sc["L"]))
    rng = np.random.default_rng(nel)
    _, _, tb, tc, _ = o.mp2()
    tb = tb + 1e-3 * rng.standard_normal(tb.shape)
    tc = tc + 1e-3 * rng.standard_normal(tc.shape)
    for mask in (4, 8, 16, 31):
        ga, gb = o.ccd_g2(tb, tc, mask)
        (ha, hb), counts, _ = profiled(lambda: ctx.ccd_g2_2ch(tb, tc, mask),
                                       lambda counts, _: any("_assemble" in k for k in counts))
        names = " ".join(counts)
        assert ("k2m_assemble" in names) == products and ("k2_assemble" in names) != products, names
        scale = max(np.abs(ga).max(), np.abs(gb).max(), 1e-300)
        assert np.abs(ha - ga).max() <= 1e-12 * scale, (mask, "abab")
        assert np.abs(hb - gb).max() <= 1e-12 * scale, (mask, "abba")


def test_one_context_through_the_forms():
    """One and two sets of integrals and the loops in turn on one context: each selection's values
    are those of a context of its own, bit for bit."""
    names = ["exchange ladders none", "short range", "one term with an excluded integral", "exchange ladders none",
             "direct ladders none", "short range"]
    o = _setup(30, 6, ONE, -1)
    sc = o.scalars()
    system = (o.nocc, sc["L"], sc["madelung"], o.eigen(), o.nvec())
    sd = _screening(2 * o.nocc, sc["L"])
    _, _, tb, tc, _ = o.mp2()
    ctx = Context(*system)
    for name in names:
        ctx.set_eri(FORMS[name][0], safe_eri=True, screening=sd)
        own = Context(*system)
        own.set_eri(FORMS[name][0], safe_eri=True, screening=sd)
        for x, y in zip(ctx.ccd_g2_2ch(tb, tc, 31), own.ccd_g2_2ch(tb, tc, 31)):
            assert np.array_equal(x, y), name


@pytest.mark.parametrize("nel,cut", [(2, 3), (14, 5)])
def test_a_repeated_selection_is_not_made_again(nel, cut):
    """A second residual with the same integrals uploads the amplitudes and nothing else; a new selection,
    and the old one after it, are taken up."""
    o = _setup(nel, cut, ONE)
    sc = o.scalars()
    ctx = Context(o.nocc, sc["L"], sc["madelung"], o.eigen(), o.nvec())
    sd = _screening(2 * o.nocc, sc["L"])
    _, _, tb, tc, _ = o.mp2()
    ctx.set_eri(ONE, safe_eri=True, screening=sd)
    first = ctx.ccd_g2_2ch(tb, tc, 31)

    def calls():
        out, counts, _ = profiled(lambda: ctx.ccd_g2_2ch(tb, tc, 31))
        return out, counts["cudaMemcpyAsync"], counts["cudaLaunchKernel"]

    again, copies, launches = calls()
    assert copies == 4   # two arrays up, two down
    ctx.set_eri(ONE, safe_eri=True, screening=2 * sd)
    other, more_copies, more_launches = calls()
    assert more_copies == copies + 1 and more_launches == launches + 1   # the tables and the weights
    ctx.set_eri(ONE, safe_eri=True, screening=sd)
    back = ctx.ccd_g2_2ch(tb, tc, 31)
    for x, y, z, w in zip(first, again, back, other):
        assert np.array_equal(x, y) and np.array_equal(x, z) and not np.array_equal(x, w)


def test_a_first_call_costs_little_more_than_the_next():
    """The lists of the products follow from sorted momenta: the first two-channel residual of an N=114
    context (57 occupied orbitals) takes about the time of the second.  Compared with every pair,
    2.2 times; best of four contexts, against half as much again."""
    import time

    from uegccd_b200 import heg

    h = heg.Heg(heg.default_input(nelectron=114, maxkpoint=50, rsmin=1.0, rsmax=1.0, fcut=(500 / 57) ** (2.0 / 3.0)))
    took = [[], []]
    for system in h.twist_systems(np.random.default_rng(2).random((4, 3)) - 0.5)[0]:
        ctx = Context(*system)
        _, _, tb, tc = ctx.mp2()
        for k in range(2):
            t0 = time.perf_counter()
            ctx.ccd_g2_2ch(tb, tc, 31)
            took[k].append(time.perf_counter() - t0)
    assert min(took[0]) <= 1.5 * min(took[1]), took
