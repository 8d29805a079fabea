"""Systems with few occupied orbitals and thousands of plane waves: one system's work has to reach more
than a few SMs, and its sums are the reference's at the edges of their ranges."""
import math

import numpy as np
import pytest

from profiled import profiled

pytestmark = pytest.mark.gpu

SMS, SM_SHARED = 148, 228 * 1024   # an SM's shared memory, of which each CTA takes 1 KB for itself


def _system(electrons, basis, seed=5):
    """The `basis` plane waves of lowest energy of a twisted system."""
    from uegccd_b200 import heg

    wide = int(1.35 * (3 * basis / (4 * math.pi)) ** (2 / 3)) + 6
    h = heg.Heg(heg.default_input(nelectron=electrons, maxkpoint=wide, rsmin=1.0, rsmax=1.0,
                                  fcut=(1.02 * basis / (electrons // 2)) ** (2.0 / 3.0)))
    h.change_twist(np.random.default_rng(seed).random(3) - 0.5)
    O, L, madelung, eigen, nvec = h.system()
    eigen, nvec = np.array(eigen), np.array(nvec)
    assert len(eigen) >= basis
    return O, L, madelung, eigen[:basis].copy(), nvec[:basis].copy()


def _kernels(call, name):
    """(grid, shared memory) of every launch of a kernel."""
    _, _, events = profiled(call, lambda _, kernels: any(name in e["name"] for e in kernels))
    return [(e["args"]["grid"][0], e["args"]["shared memory"]) for e in events if name in e["name"]]


@pytest.mark.parametrize("electrons,virtuals", [(14, 60), (14, 1024), (14, 1025), (6, 2048), (14, 2049), (4, 5000)])
def test_drpa_over_column_ranges(electrons, virtuals):
    """One CTA per occupied orbital and 1,024 virtuals; the reference's iteration in plain sums ends at
    the same amplitudes (1e-12: both stop on the same iterate, which rounding moves by less)."""
    from perf.cases import _Exact
    from uegccd_b200 import Context

    system = _system(electrons, electrons // 2 + virtuals)
    O = system[0]
    ctx = Context(*system)
    t = [None]

    def solve():
        t[0] = ctx.mp2()[1]
        assert ctx.drpa(t[0])[0] == 0

    launches = _kernels(solve, "k_drpa_sums")
    assert launches and all(g == O * -(-virtuals // 1024) for g, _ in launches), launches
    x = _Exact(system)
    p, m = x.mp2()
    (want,) = x.iterate([p + m], lambda a: (x.drpa_residual(a),), 1e-8, 2.0)
    want = x.out(want)
    assert np.abs(t[0] - want).max() <= 1e-12 * np.abs(want).max()


@pytest.mark.parametrize("electrons,basis,name", [(2, 3000, "k_ladder_fma"), (14, 3000, "k_ladder_fma"),
                                                  (54, 485, "k_ladder_mma"), (54, 1500, "k_ladder_fma")])
def test_a_short_ladder_is_spread_over_the_sms(electrons, basis, name):
    """Beside other kernels an SM takes no more of the ladder's CTAs than their share of the GPU: what
    shared memory each one holds leaves no room for another.  (Packed on the first SMs that come free, an
    iteration took up to four times as long, at random.)"""
    from uegccd_b200 import Batch

    b = Batch([_system(electrons, basis)])
    launches = _kernels(lambda: b.solve(scheme=1, ndiis=6, denom_factor=1.0, max_iter=4, raise_on_error=False), name)
    assert launches
    for grid, shared in launches:
        share = -(-grid // SMS)
        assert share <= 4
        assert SM_SHARED // (shared + 1024) == share, (grid, shared)
    b.close()
