"""Page-locked host memory of the library: what live objects hold, what downloads lock, and that
every download gives the same values whichever way it takes.

Page-locked memory shows in RssShmem of /proc/self/status.  The slack of 24 MB stands for what else
the process maps shared between two reads."""
import re

import numpy as np
import pytest

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
