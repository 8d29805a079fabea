"""The spin-adapted residual over the forms of its |q|^2 table: 16 copies in shared memory (|q|^2 below 256 and
|n|^2 below 128), one copy (|q|^2 below 1,024), global memory.

Systems with few orbitals and wide vectors: the occupied ones a cube of 27 or 64, around it the rest
of a larger cube, far away pairs of cubes that are each other's partners (blocks of up to 14 and 32
rows, ring groups of up to 27 and 64), and single orbitals that move the largest |n|^2 or |q|^2 to
either side of a line (|q|^2 = 255 and 1,023 and |n|^2 = 127 are no sums of three squares).  Against
the dense sums of perf/cases.py; tolerance 1e-12 of the largest element, as in test_gpu_parity.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cube(lo, hi, at=(0, 0, 0)):
    g = np.arange(lo, hi + 1)
    return np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3) + np.array(at)


def _system(side, far, single):
    lo, hi = (-1, 1) if side == 27 else (-1, 2)
    occ = _cube(lo, hi)
    rest = [_cube(lo - 1, hi + 1)]
    if far:
        rest += [_cube(lo, hi, (far, 0, 0)), _cube(lo, hi, (-far, 0, 0))]
    if single:
        rest.append(np.array(single))
    seen = {tuple(v) for v in occ}
    vir = [v for v in np.concatenate(rest) if not (tuple(v) in seen or seen.add(tuple(v)))]
    n = np.concatenate([occ, np.array(vir)]).astype(np.int32)
    q2 = max(int(((n - v) ** 2).sum(1).max()) for v in n)
    eigen = 0.02 * (n.astype(float) ** 2).sum(1) + np.where(np.arange(len(n)) < len(occ), -1.0, 1.0)
    return (len(occ), 6.0, 0.4, eigen, n), q2, int((n ** 2).sum(1).max())


CASES = {
    # occupied, distance of the far cubes, single orbitals; the form
    "16 copies, both at their ends": (27, 0, [(11, 2, 1), (-4, -3, -1)], "16", 254, 126),
    "|n|^2 one too large": (27, 0, [(8, 8, 0)], "1", None, 128),
    "|q|^2 one too large": (27, 0, [(8, 0, 0), (-8, 0, 0)], "1", 256, None),
    "one copy, 27": (27, 7, None, "1", None, None),
    "one copy, 64": (64, 8, None, "1", None, None),
    "one copy, at its end": (27, 0, [(15, 3, 2), (-16, -3, -3)], "1", 1022, None),
    "global, at its start": (27, 0, [(16, 0, 0), (-16, 0, 0)], "global", 1024, None),
    "global, 27": (27, 15, None, "global", None, None),
    "global, 64": (64, 16, None, "global", None, None),
    "global, the widest vectors": (27, 62, None, "global", None, None),
}


@pytest.mark.parametrize("case", CASES)
def test_residual(case):
    from perf.cases import _Exact
    from uegccd_b200 import Context

    side, far, single, form, q2want, n2want = CASES[case]
    system, q2max, n2max = _system(side, far, single)
    assert q2want in (None, q2max) and n2want in (None, n2max), (q2max, n2max)
    assert form == ("16" if q2max < 256 and n2max < 128 else "1" if q2max < 1024 else "global")
    ctx = Context(*system)
    x = _Exact(system)
    p, m = x.mp2()
    _, _, tb, _ = ctx.mp2()
    assert np.abs(tb - x.out(p)).max() <= 1e-14 * float(p.abs().max())
    for mask, kw in ((31, {}), (15, dict(xring=False)), (7, dict(ring=False, xring=False))):
        want = x.out(x.residual(p, m, **kw)[0])
        g = ctx.ccd_g2(x.out(p), mask)
        scale = np.abs(want).max()
        assert np.abs(g - want).max() <= 1e-12 * scale, (mask, np.abs(g - want).max() / scale)
