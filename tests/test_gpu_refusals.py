"""Options that the particle pass refuses are refused for any number of turns
and by prepare, with and without collective effects; nothing is tracked."""
import numpy as np
import pytest
import torch

from blond_b200 import BlondB200Error, _lib
from blond_b200.beam.beam import Beam, Proton
from blond_b200.beam.distributions import _get_dE_from_dt, bigaussian_arrays
from blond_b200.beam.profile import CutOptions, Profile
from blond_b200.engine import FusedTracker
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.trackers.tracker import RingAndRFTracker

pytestmark = pytest.mark.gpu


def _fused(S, kernel, turns=120):
    ring = Ring(6911.5, 1 / 18**2, 26e9, Proton(), turns)
    rf = RFStation(ring, [4620], [4.5e6], [0.0])
    centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
    dt, dE = bigaussian_arrays(1001, 0.4e-9, _get_dE_from_dt(ring, rf, 0.4e-9), centre, 7)
    beam = Beam(ring, len(dt), 1e10, dt=dt, dE=dE, dtype=torch.float64)
    prof = Profile(beam, CutOptions(cut_left=centre - 1.25e-9, cut_right=centre + 1.25e-9,
                                    n_slices=S))
    return FusedTracker(RingAndRFTracker(rf, beam), prof, precision="f64", kernel=kernel)


# no interpolated kick; a ring of 4 stages beside 200 KB of histogram
@pytest.mark.parametrize("S,kernel,prefetch,match", [
    (100, "stab", 0, "shared-table"), (100, "packed", 0, "packed-histogram"),
    (50_000, "plain", 4, "prefetch ring")])
def test_refused_for_any_number_of_turns(cuda, S, kernel, prefetch, match):
    fused = _fused(S, kernel)
    fused.eng.call("set_prefetch", prefetch)
    dt, dE = fused.dt.clone(), fused.dE.clone()
    for turns in (1, 2, 50, 117):
        with pytest.raises(BlondB200Error, match=match):
            fused.track(turns)
    with pytest.raises(BlondB200Error, match=match):
        fused.eng.call("prepare", _lib.stream())
    assert torch.equal(fused.dt, dt) and torch.equal(fused.dE, dE)
    # and with options that fit the same object tracks
    fused.eng.call("set_kernel", 1)
    fused.eng.call("set_prefetch", 0)
    fused.eng.call("prepare", _lib.stream())
    fused.track(3)
    fused.check()
    assert not torch.equal(fused.dt, dt)
    assert np.isfinite(fused.dt.cpu().numpy()).all()
