"""The workspace of the two-channel matrix products is one for a batch, and gives way: what a batch
solves without it, it solves under a memory limit that leaves no room for it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIIS = dict(scheme=1, ndiis=6, denom_factor=1.0)
TWO = dict(do_ring=1, do_xring=0)   # rings without crossed rings: both channels iterated
MB = 1 << 20


def _systems(sizes, seed=11):
    from uegccd_b200 import heg

    rng = np.random.default_rng(seed)
    out = []
    for electrons, basis in sizes:
        h = heg.Heg(heg.default_input(nelectron=electrons, maxkpoint=50, rsmin=1.0, rsmax=1.0,
                                      fcut=(basis / (electrons // 2)) ** (2.0 / 3.0)))
        out += h.twist_systems(rng.random((1, 3)) - 0.5)[0]
    return out


def _live():
    from uegccd_b200 import _capi

    held, cached = _capi.memory_info()
    return held - cached


def _solve(b, **kw):
    rc, _, res = b.solve(**TWO, **kw)
    assert rc == 0
    return [(r["ecorr"], r["niter"], r["ndiis"]) for r in res], [t.copy() for t in b.all_amplitudes()]


@pytest.mark.parametrize("options", [{}, DIIS], ids=["replay", "diis"])
def test_batch_under_a_limit_that_holds_the_loops(options):
    """Eight N=54 systems (29 MB each, the products' workspace 21 MB) under the bytes the batch takes
    when a core orbital rules the products out: every system solves, with its whole history."""
    from uegccd_b200 import Batch, _capi

    systems = _systems([(54, 485)] * 8)
    b = Batch(systems)
    want, t = _solve(b, **options)
    b.close()
    _capi.trim_cache()
    base = _live()
    b = Batch(systems)
    _solve(b, core_n=1, max_iter=40, **options)
    loops = _live() - base
    b.close()
    _capi.trim_cache()
    try:
        _capi.set_memory_limit(_live() + loops)
        b = Batch(systems)
        got, u = _solve(b, **options)
        again, _ = _solve(b, **options)
        b.close()
    finally:
        _capi.set_memory_limit(0)
    for x in (got, again):
        assert [k[2] for k in x] == [k[2] for k in want]
        np.testing.assert_allclose([k[0] for k in x], [k[0] for k in want], rtol=1e-12)
    for x, y in zip(t, u):
        assert np.abs(x - y).max() <= 1e-10


def test_one_workspace_serves_systems_of_all_sizes():
    """Systems of four sizes, large and small in turn, twice: each has the bits it has in a batch of its
    own, and the batch holds one workspace over what it holds without (21 MB; one chunk of 64 MB)."""
    from uegccd_b200 import Batch, _capi

    systems = _systems([(54, 485), (14, 57), (38, 247), (54, 400), (2, 40), (54, 485)])
    want = []
    for s in systems:
        b = Batch([s])
        r, t = _solve(b)
        want.append((r[0], t[0]))
        b.close()
    _capi.trim_cache()
    base = _live()
    b = Batch(systems)
    for _ in range(2):
        r, t = _solve(b)
        for k, (w, x) in enumerate(want):
            assert r[k] == w, k
            assert np.array_equal(t[k], x), k
    held = _live() - base
    b.close()
    _capi.trim_cache()
    b = Batch(systems)
    b.solve(**TWO, core_n=1, max_iter=3)
    b.all_amplitudes()
    loops = _live() - base
    b.close()
    assert held <= loops + 32 * MB, (held / MB, loops / MB)


def test_idle_workspace_gives_way_to_a_history():
    """A context's residual takes the workspace; its solve then finds room for 13 history vectors of
    both channels under a limit that holds them or the workspace, not both."""
    from uegccd_b200 import Context, _capi

    _capi.trim_cache()   # a cached chunk may be larger than the request it serves
    ctx = Context(*_systems([(54, 485)])[0])
    _, aa, ab, ba = ctx.mp2()
    ctx.drpa_g2(ab, 15)   # the state of both channels, without the workspace
    history = 4 * 13 * ab.nbytes
    try:
        _capi.set_memory_limit(_live() + history + MB)
        g = ctx.ccd_g2_2ch(ab, ba, 15)
        rc, r, _, _ = ctx.ccd(aa, ab, ba, **TWO, scheme=1, ndiis=13, denom_factor=1.0)
        assert rc == 0 and r["ndiis"] == 13
        h = ctx.ccd_g2_2ch(*ctx.mp2()[2:4], 15)   # by the loops where there is no room
    finally:
        _capi.set_memory_limit(0)
    again = ctx.ccd_g2_2ch(*ctx.mp2()[2:4], 15)
    for x, y, z in zip(g, h, again):
        assert np.array_equal(x, z)
        assert np.abs(x - y).max() <= 1e-12 * np.abs(x).max()


def test_contexts_share_what_room_there_is():
    """Residuals of two live contexts in turn under limits with room for no, one and both workspaces."""
    from uegccd_b200 import Context, _capi

    ctx = [Context(*s) for s in _systems([(54, 485), (54, 485)], seed=5)]
    t = [c.mp2()[2:4] for c in ctx]
    want = [c.ccd_g2_2ch(*x, 15) for c, x in zip(ctx, t)]
    try:
        for room in (0, 24 * MB, 48 * MB):
            _capi.set_memory_limit(0)
            _capi.trim_cache()   # the idle workspaces go back
            _capi.set_memory_limit(_live() + room)
            for _ in range(2):
                for c, x, w in zip(ctx, t, want):
                    for a, r in zip(c.ccd_g2_2ch(*x, 15), w):
                        assert np.abs(a - r).max() <= 1e-12 * np.abs(r).max()
    finally:
        _capi.set_memory_limit(0)
    for c, x, w in zip(ctx, t, want):
        for a, r in zip(c.ccd_g2_2ch(*x, 15), w):
            assert np.array_equal(a, r)
