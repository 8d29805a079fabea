"""dRPA from the particle-hole sums (k_drpa_sums): replay solves of a ragged batch against the
oracle -- one occupied orbital, fewer virtuals than a CTA has threads, more than a CTA has,
with and without mosaics and rings -- and the same batch solved twice.  Tolerances as in
test_gpu_parity.py: the oracle's iteration count, energies within 1e-11 Ha."""
import numpy as np
import pytest

from oracle.oracle import Oracle, parse_input_text

pytestmark = pytest.mark.gpu

# electrons, momentum cutoff: (1 occupied, 18 virtuals), (7, 50), (19, 321: two passes a thread)
SIZES = ((2, 3), (14, 5), (38, 17))


def _oracle(nel, cut, twist, mosaic, ring):
    v = parse_input_text("")
    v.update({"# Electrons": str(nel), "Momentum Cutoff": str(cut), "Do Mosaics": mosaic, "Do Rings": ring})
    o = Oracle(v)
    o.change_twist(twist)
    return o


@pytest.mark.parametrize("mosaic,ring", [("T", "T"), ("F", "T"), ("T", "F")])
def test_ragged_drpa_batch_matches_oracle(mosaic, ring):
    from uegccd_b200 import Batch

    os_ = [_oracle(n, c, (0.1 + 0.03 * k, -0.2, 0.3), mosaic, ring) for k, (n, c) in enumerate(SIZES)]
    systems = []
    for o in os_:
        sc = o.scalars()
        systems.append((o.nocc, sc["L"], sc["madelung"], o.eigen(), o.nvec()))
    b = Batch(systems)
    runs = [b.solve(drpa=True, do_mosaic=int(mosaic == "T"), do_ring=int(ring == "T")) for _ in range(2)]
    amps = [b.amplitudes(s) for s in range(len(systems))]
    for s, o in enumerate(os_):
        _, ta, _, _, _ = o.mp2()
        st, _, _ = o.drpa(ta)
        for _, _, res in runs:   # the second solve starts from the MP2 amplitudes again
            assert res[s]["niter"] == st.niter
            assert abs(res[s]["ecorr"] - st.ecorr) < 1e-11
            assert abs(res[s]["ecorr_sosex"] - st.ecorr_sosex) < 1e-11
        assert np.abs(amps[s] - ta).max() < 1e-11
