"""The kernels of the spin-adapted solve at the sizes where their tiles can go wrong, against the
oracle and against each other.

Residual terms, one system each (electrons, momentum cutoff): one occupied orbital; one with 6,000
columns in its only block, many passes of every column tile, |n|^2 beyond the byte that the
16-copy Coulomb table needs; blocks of up to 4, 8, 14, 16 and 29 rows i <= j (both forms of the ladder,
one and two of its row tiles); ring pairs of up to 7, 15, 23, 31, 45 and 57 rows (each class of
k_rings).  Tolerance: 1e-12 of the largest element, as in test_gpu_parity.py.
"""
import threading

import numpy as np
import pytest

from oracle.oracle import Oracle, parse_input_text

pytestmark = pytest.mark.gpu

DIIS = dict(scheme=1, ndiis=6, denom_factor=1.0)


def _oracle(nel, cut, twist=(0.11, -0.23, 0.31)):
    v = parse_input_text("")
    v.update({"# Electrons": str(nel), "Momentum Cutoff": str(cut), "rSMin": "1.0", "rSMax": "1.0"})
    if cut > 100:
        v["fcut"] = "330"   # 6,000 orbitals for one occupied
    o = Oracle(v)
    o.change_twist(twist)
    return o


def _system(o):
    sc = o.scalars()
    return (o.nocc, sc["L"], sc["madelung"], o.eigen(), o.nvec())


def _twists(count, electrons=54, basis=485):
    from uegccd_b200 import heg

    h = heg.Heg(heg.default_input(nelectron=electrons, maxkpoint=50, rsmin=1.0, rsmax=1.0,
                                  fcut=(basis / (electrons // 2)) ** (2.0 / 3.0)))
    return h.twist_systems(np.random.default_rng(5).random((count, 3)) - 0.5)[0]


@pytest.mark.parametrize("nel,cut", [(2, 3), (2, 140), (14, 5), (30, 6), (46, 9), (54, 10), (62, 11), (90, 14), (114, 14)])
def test_residual_terms_over_sizes(nel, cut):
    from uegccd_b200 import Context

    o = _oracle(nel, cut, (0.0, 0.0, 0.0) if nel in (54, 114) else (0.11, -0.23, 0.31))
    _, _, tb, tc, _ = o.mp2()
    ctx = Context(*_system(o))
    for mask in (1, 2, 4, 8, 16, 31):
        ga, _ = o.ccd_g2(tb, tc, mask)
        g = ctx.ccd_g2(tb, mask)
        scale = np.abs(ga).max()
        assert np.abs(g - ga).max() <= 1e-12 * scale, (mask, np.abs(g - ga).max(), scale)


@pytest.mark.parametrize("ndiis", [2, 3, 7, 8, 16])
def test_history_depths_reach_the_fixed_point(ndiis):
    """Both instances of the update's push (up to 7 vectors, up to 16) and the elimination of every
    depth: the tight energy of the reference's iteration.  Tolerance as in test_gpu_diis.py."""
    from uegccd_b200 import Context

    o = _oracle(14, 5)
    _, ta, tb, tc, _ = o.mp2()
    st, _, _ = o.ccd(ta, tb, tc, tol=1e-12)
    ctx = Context(*_system(o))
    _, ga, gb, gc = ctx.mp2()
    rc, r, _, _ = ctx.ccd(ga, gb, gc, **dict(DIIS, ndiis=ndiis), tol=1e-12)
    assert rc == 0
    assert abs(r["ecorr"] - st.ecorr) < 1e-10, (r["ecorr"], st.ecorr)
    assert np.abs(gb - tb).max() < 1e-10


@pytest.mark.parametrize("count", [2, 45])
def test_streams_of_a_residual_give_the_same_bits(count):
    """The terms beside each other (2 systems), the ring classes beside each other (45: 0.22 M packed
    amplitudes each, together more than 9 M) and one stream (sampled iterations under the kernel timers): the sums are ordered,
    so nothing may change."""
    from uegccd_b200 import Batch

    b = Batch(_twists(count))
    runs = []
    for timers in (0, 1, 0):
        b.set_profiling(bool(timers))
        _, e2, res = b.solve(**DIIS)
        runs.append((np.array([r["ecorr"] for r in res]), [r["niter"] for r in res], b.amplitudes(0)))
    b.close()
    for e, n, t in runs[1:]:
        assert np.array_equal(e, runs[0][0]) and n == runs[0][1] and np.array_equal(t, runs[0][2])


def test_kept_graphs_follow_options_and_buffers():
    """A mixed solve, an FP64 one with a deeper history (its buffers move) and the mixed one again;
    a solve that stops at its start in between leaves nothing behind."""
    from uegccd_b200 import Batch

    b = Batch(_twists(3, electrons=14, basis=60))
    mixed = dict(DIIS, ndiis=4, precision=1)

    def run(**kw):
        _, _, res = b.solve(**kw)
        return [(r["ecorr"], r["niter"]) for r in res], b.amplitudes(1)

    e0, t0 = run(**mixed)
    f0, u0 = run(**dict(DIIS, ndiis=12))
    assert all(n == 1 for _, n in run(**DIIS, tol=1e3)[0])
    e1, t1 = run(**mixed)
    f1, u1 = run(**dict(DIIS, ndiis=12))
    b.close()
    assert e0 == e1 and np.array_equal(t0, t1)
    assert f0 == f1 and np.array_equal(u0, u1)


def test_downloads_of_every_size():
    """A context's amplitudes through the shared page-locked buffers: 3 x 0.03, 3 x 0.66 and 3 x 28 MB
    (one thread, all cores), a residual of 28 MB (straight), from three threads at once; the batch's
    packed amplitudes unpacked on their own are the reference."""
    from uegccd_b200 import Batch, Context

    systems = [_twists(1, n, m)[0] for n, m in ((14, 60), (38, 247), (114, 1140))]
    want, errors = [], []
    for s in systems:
        b = Batch([s])
        b.mp2()
        want.append(b.amplitudes(0))
        b.close()

    def work(s, w):
        try:
            ctx = Context(*s)
            g = None
            for _ in range(3):
                _, _, tab, tba = ctx.mp2()
                assert np.array_equal(tab, w)
                r = ctx.ccd_g2(tab)
                assert g is None or np.array_equal(r, g)
                g = r
        except Exception as e:   # an assertion of a thread has to reach the test
            errors.append(repr(e))

    th = [threading.Thread(target=work, args=a) for a in zip(systems, want)]
    for x in th:
        x.start()
    for x in th:
        x.join()
    assert not errors, errors
