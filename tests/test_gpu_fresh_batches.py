"""What a program that makes a batch for every step pays for beside the batch itself: streams,
events, page-locked and device memory come from the batches before."""
import threading

import numpy as np
import pytest

from profiled import profiled

pytestmark = pytest.mark.gpu

DIIS = dict(scheme=1, ndiis=6, denom_factor=1.0)


def _systems(count, electrons, basis, seed=3):
    from uegccd_b200 import heg

    h = heg.Heg(heg.default_input(nelectron=electrons, maxkpoint=50, rsmin=1.0, rsmax=1.0,
                                  fcut=(basis / (electrons // 2)) ** (2.0 / 3.0)))
    return h.twist_systems(np.random.default_rng(seed).random((count, 3)) - 0.5)[0]


def _step(systems, drpa):
    from uegccd_b200 import Batch

    b = Batch(systems)
    _, e2, res = b.solve(drpa=drpa, **({} if drpa else DIIS))
    out = list(e2), [r["ecorr"] for r in res], [t.copy() for t in b.all_amplitudes()]
    b.close()
    return out


@pytest.mark.parametrize("drpa", [False, True], ids=["ccd", "drpa"])
@pytest.mark.parametrize("count,electrons,basis", [(3, 14, 42), (10, 38, 228)])
def test_a_batch_takes_over_what_the_last_one_used(count, electrons, basis, drpa):
    """A second batch makes its own stream and nothing more, dRPA (which has no side streams) from the
    first one on; and its values are the first one's."""
    from uegccd_b200 import _capi

    systems = _systems(count, electrons, basis)
    _capi.trim_cache()
    counts, outs = [], []
    for _ in range(2):
        out, c, _ = profiled(lambda: _step(systems, drpa))
        outs.append(out)
        counts.append(c)
    assert counts[1]["cudaGraphLaunch"] > 0
    for c in counts[0 if drpa else 1:]:
        assert c["cudaStreamCreateWithFlags"] == 1 and c["cudaStreamDestroy"] == 1, c
    assert "cudaHostAlloc" not in counts[1] and "cudaFreeHost" not in counts[1], counts[1]
    assert "cudaMalloc" not in counts[1] and "cudaFree" not in counts[1], counts[1]
    (a2, a, ta), (b2, b, tb) = outs
    assert a2 == b2 and a == b and all(np.array_equal(x, y) for x, y in zip(ta, tb))


def test_side_streams_of_many_threads_and_live_batches():
    """Six threads make, solve and release batches of two sizes while other batches stay alive, and
    the idle sets are given up in between: the values are those of one batch alone."""
    from uegccd_b200 import Batch, _capi

    sets = [_systems(3, 14, 60), _systems(2, 54, 485)]
    want = [_step(s, False) for s in sets]
    live = [Batch(s) for s in sets]
    for b in live:
        b.solve(**DIIS)
    errors = []

    def work(k):
        try:
            for rep in range(3):
                q = (k + rep) % 2
                got = _step(sets[q], False)
                assert got[0] == want[q][0] and got[1] == want[q][1]
                assert all(np.array_equal(x, y) for x, y in zip(got[2], want[q][2]))
                if k == 0:
                    _capi.trim_cache()
        except Exception as e:   # an assertion of a thread has to reach the test
            errors.append(repr(e))

    th = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for x in th:
        x.start()
    for x in th:
        x.join()
    assert not errors, errors
    for b, w in zip(live, want):
        assert [r["ecorr"] for r in b.solve(**DIIS)[2]] == w[1]
        b.close()


def test_reported_launch_shapes_are_those_launched():
    """ring_threads and launch_shapes against the profile of a solve with ring groups of all sizes."""
    import re

    from uegccd_b200 import Batch

    b = Batch(_systems(1, 114, 1140))
    b.solve(**DIIS)

    def threads(events):
        """Rows of group 1 in eights -> threads."""
        found = ((re.search(r"k_rings<\w+, (\d)>", e["name"]), e["args"]["block"][0]) for e in events)
        return {int(m.group(1)): n for m, n in found if m}

    _, _, events = profiled(lambda: b.solve(**DIIS), lambda _, kernels: len(threads(kernels)) == 6)
    sizes = threads(events)
    assert sorted(sizes) == [1, 2, 3, 4, 6, 8]
    of = {8: [1], 4: [2], 2: [3, 4], 1: [6, 8]}   # pairs a CTA
    shapes = b.launch_shapes()
    assert b.ring_threads() == shapes["ring_threads"] == [max(sizes[n] for n in of[k]) for k in (8, 4, 2, 1)]
    stage = {e["args"]["block"][0] for e in events if "k_ring_stage" in e["name"]}
    assert stage == {shapes["stage_threads"]}
    b.close()


@pytest.mark.parametrize("options", [dict(), DIIS, dict(DIIS, precision=1), dict(drpa=True), dict(do_ring=1, do_xring=0)],
                         ids=["replay", "diis", "mixed", "drpa", "two channels"])
@pytest.mark.parametrize("count,electrons,basis", [(2, 54, 485), (3, 14, 60)])
def test_reported_launches_are_those_made(count, electrons, basis, options):
    """kernel_launches of a solve against the kernels of its profile: all but the MP2 start's two (or
    three, with dRPA's T2aaaa), which are not the solve's."""
    from uegccd_b200 import Batch

    b = Batch(_systems(count, electrons, basis))
    b.solve(**options)
    two, made = "do_xring" in options, [0]
    start = 0 if two else 3 if options.get("drpa") else 2

    def solve():
        reported[:] = [r["kernel_launches"] for r in b.solve(**options)[2]]

    def complete(counts, _):
        # with two channels one count a system; the batch's own kernels around the solves are not counted
        kernels = {k: n for k, n in counts.items() if "uegccd::" in k and not (two and "::k_" in k)}
        made[0] = sum(kernels.values()) - start
        return made[0] == want()

    def want():
        return sum(reported) if two else reported[0]

    reported = []
    profiled(solve, complete)
    assert made[0] == want(), (made[0], reported)
    b.close()
