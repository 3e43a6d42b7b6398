"""Several turns per launch with profiles whose histogram leaves room for fewer
turns' constants, or none, in a block's shared memory: the same bits as the same
turns one call at a time.  On a B200 54000 slices leave 27 turns to the launch
that deposits, 57700 one, 57719 and 65536 none (a single turn deposits) and
100000 take the global histogram in either way."""
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


def _fused(n, S, turns, precision, kernel, half):
    ring = Ring(6911.5, 1 / 18**2, 26e9 + 1e4 * np.arange(turns + 1), Proton(), turns)
    rf = RFStation(ring, [4620], [4.5e6], [0.0])
    centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
    dt, dE = bigaussian_arrays(n, 0.4e-9, _get_dE_from_dt(ring, rf, 0.4e-9), centre, 7)
    beam = Beam(ring, n, 1e10, dt=dt, dE=dE, dtype=torch.float64)
    prof = Profile(beam, CutOptions(cut_left=centre - half, cut_right=centre + half, n_slices=S))
    return FusedTracker(RingAndRFTracker(rf, beam), prof, precision=precision, kernel=kernel,
                        energy_unit=1.0)


@pytest.mark.parametrize("kernel", ["plain", "tma"])
@pytest.mark.parametrize("precision", ["f64", "f32p64", "q32p64"])
# windows of 2.5 ns, and of 4 us: the whole bunch in a few slices
@pytest.mark.parametrize("S,half", [(54000, 1.25e-9), (57700, 1.25e-9), (57719, 1.25e-9),
                                    (65536, 2e-6), (100000, 1.25e-9)])
def test_same_bits_as_single_turns(cuda, precision, kernel, S, half):
    steps = (2, 28, 65, 92)
    many = _fused(20001, S, sum(steps) + 1, precision, kernel, half)
    single = _fused(20001, S, sum(steps) + 1, precision, kernel, half)
    for turns in steps:
        many.track(turns)
        for _ in range(turns):
            single.track(1)
        assert torch.equal(many.dt, single.dt)
        assert torch.equal(many.dE, single.dE)
        assert torch.equal(many.profile_tensor(), single.profile_tensor())
        assert many.profile_tensor().sum() > 19000
    many.track(1)
    single.track(1)
    many.check()
    assert torch.equal(many.dt, single.dt) and torch.equal(many.dE, single.dE)
