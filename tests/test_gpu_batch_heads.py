"""Batched beams against the single-beam engine where the two take different
heads: the same voltages within rounding, the counts and the kick as they follow.

Bars: the voltages come from the same profiles by two transforms, each within
2e-14 of max|V| (test_gpu_head_accuracy.py gives the convolution's bound, smaller
for these resonators): 4e-14.  The energies then differ by that share of the
largest voltage, and by the rounding of an energy.
"""
import numpy as np
import pytest
import torch

from blond_b200.batch import BatchTracker
from blond_b200.beam.beam import Beam, Proton
from blond_b200.beam.distributions import bigaussian_arrays
from blond_b200.beam.profile import CutOptions, Profile
from blond_b200.engine import FusedTracker
from blond_b200.impedances.impedance import InducedVoltageFreq, TotalInducedVoltage
from blond_b200.impedances.impedance_sources import Resonators
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.trackers.tracker import RingAndRFTracker

pytestmark = pytest.mark.gpu


def _objects(n, S, seed):
    ring = Ring(6911.5, 1 / 18**2, 26e9, Proton(), 3)
    rf = RFStation(ring, [4620], [4.5e6], [0.0])
    centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
    dt, dE = bigaussian_arrays(n, 0.4e-9, 1e8, centre, seed)
    beam = Beam(ring, n, 1e10, dt=dt, dE=dE, dtype=torch.float64)
    prof = Profile(beam, CutOptions(cut_left=centre - 1.25e-9, cut_right=centre + 1.25e-9,
                                    n_slices=S))
    tiv = TotalInducedVoltage(beam, prof, [InducedVoltageFreq(
        beam, prof, [Resonators([2e5, 1e5], [200e6, 1.4e9], [100.0, 3000.0])])])
    return RingAndRFTracker(rf, beam), prof, tiv


# single / batch: convolution / mixed radix (9000, 12000), padded transform /
# mixed radix (14000), 16-CTA / general transform (8192), convolution / power of
# two (64 of 512); convolution both, with other tiles per block (150 of 64, 37 of
# 400, 8 of 4096): equal bits
@pytest.mark.parametrize("B,S,same", [(2, 9000, False), (3, 12000, False), (2, 14000, False),
                                      (3, 8192, False), (64, 512, False), (150, 64, True),
                                      (37, 400, True), (8, 4096, True)])
def test_same_voltages_as_single_beams(cuda, B, S, same):
    batch = BatchTracker([_objects(3000 + b, S, b) for b in range(B)], precision="f64")
    singles = [FusedTracker(*_objects(3000 + b, S, b), precision="f64")
               for b in range(0, B, max(1, B // 5))]
    batch.track(1)
    V, p = batch.induced_voltages_tensor(), batch.profiles_tensor()
    for b, one in zip(range(0, B, max(1, B // 5)), singles):
        one.track(1)
        v = one.induced_voltage_tensor()
        top = float(v.abs().max())
        assert top > 0
        assert float((V[b] - v).abs().max()) <= 4e-14 * top
        if same:
            assert torch.equal(V[b], v)
            assert torch.equal(batch.coordinates(b)[1], one.dE)
        assert torch.equal(p[b], one.profile_tensor())
        dE = batch.coordinates(b)[1]
        eps = np.finfo(float).eps
        assert float((dE - one.dE).abs().max()) <= 1e-13 * top + 2 * eps * float(dE.abs().max())
