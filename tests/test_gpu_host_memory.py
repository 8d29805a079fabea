"""Page-locked host memory of the library: what live objects hold, what downloads lock, and that
every download gives the same values whichever way it takes.

Page-locked memory shows in RssShmem of /proc/self/status.  The slack of 24 MB stands for what else
the process maps shared between two reads."""
import re

import numpy as np
import pytest

from profiled import profiled

pytestmark = pytest.mark.gpu

MB = 1 << 20
SLACK = 24 * MB


def _locked():
    with open("/proc/self/status") as f:
        return int(re.search(r"RssShmem:\s+(\d+)", f.read()).group(1)) * 1024


def _systems(count, electrons, basis):
    from uegccd_b200 import heg

    h = heg.Heg(heg.default_input(nelectron=electrons, maxkpoint=50, rsmin=1.0, rsmax=1.0,
                                  fcut=(basis / (electrons // 2)) ** (2.0 / 3.0)))
    return h.twist_systems(np.random.default_rng(7).random((count, 3)) - 0.5)[0]


def test_live_contexts_hold_no_download_buffer():
    """Four live N=114 contexts, each with an MP2 download (three arrays of 28 MB) before its solve:
    one download buffer among them, and it is idle again after each call."""
    from uegccd_b200 import Context, _capi

    systems = _systems(4, 114, 1140)
    _capi.trim_cache()
    base, live = _locked(), []
    for s in systems:
        c = Context(*s)
        _, aa, ab, ba = c.mp2()
        c.ccd(aa, ab, ba, max_iter=3)
        live.append(c)
    arrays = 3 * ab.nbytes
    assert _locked() - base <= arrays + SLACK, ((_locked() - base) / MB, arrays / MB)
    _capi.trim_cache()
    assert _locked() - base <= SLACK, (_locked() - base) / MB


def _host_allocs(call):
    """How often a call locks host memory anew."""
    _, counts, _ = profiled(call)
    assert "cudaMemcpyAsync" in counts
    return counts.get("cudaHostAlloc", 0)


@pytest.mark.parametrize("count,electrons,basis", [(2, 14, 60), (30, 54, 485), (22, 114, 1140)])
def test_batch_downloads_into_ordinary_memory(count, electrons, basis):
    """Into a new array: 0.04 MB, 80 MB (three pieces) and 590 MB (more than is kept locked).  A
    second download locks nothing, and both have the values of the solves one by one."""
    from uegccd_b200 import Batch, _capi

    b = Batch(_systems(count, electrons, basis))
    b.mp2()
    _capi.trim_cache()
    base = _locked()
    first = b.all_amplitudes()
    kept = _locked() - base
    assert kept <= 96 * MB + SLACK, kept / MB
    got = []
    assert _host_allocs(lambda: got.append(b.all_amplitudes())) == 0
    for s in range(b.n):
        want = b.amplitudes(s)
        np.testing.assert_array_equal(first[s], want)
        np.testing.assert_array_equal(got[0][s], want)
    b.close()


def test_many_threads_download_at_once():
    """Eight threads with three arrays of 28 MB each ask for more than may be locked (8 x 84 MB):
    those that find none left take the driver's copies, with the same values."""
    import threading

    from uegccd_b200 import Context, _capi

    system = _systems(1, 114, 1140)[0]
    contexts = [Context(*system) for _ in range(8)]
    want = contexts[0].mp2()
    _capi.trim_cache()
    base, errors, most = _locked(), [], [0]

    def work(c):
        try:
            for _ in range(2):
                got = c.mp2()
                most[0] = max(most[0], _locked() - base)
                assert got[0] == want[0]
                for x, y in zip(got[1:], want[1:]):
                    assert np.array_equal(x, y)
        except Exception as e:   # an assertion of a thread has to reach the test
            errors.append(repr(e))

    th = [threading.Thread(target=work, args=(c,)) for c in contexts]
    for x in th:
        x.start()
    for x in th:
        x.join()
    assert not errors, errors
    assert most[0] <= 512 * MB + SLACK, most[0] / MB


def test_small_batch_downloads_are_one_copy():
    """Below 8 MB the driver's own staging is the faster way: a download of 2.0 MB into ordinary memory
    is one copy to pageable memory, one of 10.7 MB comes through page-locked memory."""
    from uegccd_b200 import Batch

    for count, electrons, basis, key in ((3, 38, 247, "Pageable"), (4, 54, 485, "Pinned")):
        b = Batch(_systems(count, electrons, basis))
        b.mp2()
        first = b.all_amplitudes()
        again, counts, _ = profiled(b.all_amplitudes, lambda counts, _: any("Memcpy DtoH" in k for k in counts))
        copies = [k for k in counts if "Memcpy DtoH" in k]
        assert copies == [f"Memcpy DtoH (Device -> {key})"], copies
        for x, y in zip(first, again):
            np.testing.assert_array_equal(x, y)
        b.close()
