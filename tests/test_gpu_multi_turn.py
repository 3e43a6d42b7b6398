"""Several turns per launch (a beam without collective effects): the same
bits as the same turns one call at a time, which run one pass per turn."""
import numpy as np
import pytest
import torch

from blond_b200.beam.beam import Beam, Proton
from blond_b200.beam.distributions import _get_dE_from_dt, bigaussian_arrays
from blond_b200.beam.profile import CutOptions, Profile
from blond_b200.engine import FusedTracker
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.trackers.tracker import RingAndRFTracker

pytestmark = pytest.mark.gpu


def _fused(n, S, turns, precision, solver, n_rf):
    ring = Ring(6911.5, 1 / 18**2, 26e9 + 1e4 * np.arange(turns + 1), Proton(), turns)
    rf = RFStation(ring, [4620, 18480, 9240][:n_rf], [4.5e6, 4.5e5, 1e5][:n_rf],
                   [0.0, np.pi, 0.3][:n_rf], n_rf=n_rf)
    centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
    dt, dE = bigaussian_arrays(n, 0.4e-9, _get_dE_from_dt(ring, rf, 0.4e-9), centre, 7)
    beam = Beam(ring, n, 1e10, dt=dt, dE=dE, dtype=torch.float64)
    prof = Profile(beam, CutOptions(cut_left=centre - 1.25e-9, cut_right=centre + 1.25e-9,
                                    n_slices=S))
    return FusedTracker(RingAndRFTracker(rf, beam, solver=solver), prof, precision=precision,
                        kernel="plain", energy_unit=1.0)


# launches hold at most 64 turns: edges at 64 and 65; 60000 slices deposit
# into the global histogram
@pytest.mark.parametrize("precision", ["f64", "f32p64", "q32p64"])
@pytest.mark.parametrize("n,S,turns,solver,n_rf", [
    (1, 10, 2, "simple", 1), (2, 10, 64, "legacy", 1), (333, 100, 65, "exact", 2),
    (70001, 1000, 3, "simple", 2), (310003, 100, 131, "simple", 1),
    (20001, 60000, 5, "legacy", 3), (20000, 16384, 70, "exact", 1)])
def test_same_bits_as_single_turns(cuda, precision, n, S, turns, solver, n_rf):
    many = _fused(n, S, turns + 2, precision, solver, n_rf)
    single = _fused(n, S, turns + 2, precision, solver, n_rf)
    many.track(turns)
    for _ in range(turns):
        single.track(1)
    # and on from there, one more turn each way
    many.track(1)
    single.track(1)
    many.check()
    assert torch.equal(many.dt, single.dt)
    assert torch.equal(many.dE, single.dE)
    assert torch.equal(many.profile_tensor(), single.profile_tensor())
