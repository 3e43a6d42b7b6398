"""The packed pass's register pipeline gives the packed pass's bits.  Only the
autotuner sets it (it wins for FP64 at 2^16 slices on a B200); where it picks
another pass there is nothing to compare and the case is skipped.  Odd and
small counts leave threads with none, one or two pairs."""
import numpy as np
import pytest
import torch

from blond_b200.beam.beam import Beam, Proton
from blond_b200.beam.distributions import _get_dE_from_dt, bigaussian_arrays
from blond_b200.beam.profile import CutOptions, Profile
from blond_b200.engine import FusedTracker
from blond_b200.impedances.impedance import InducedVoltageFreq, TotalInducedVoltage
from blond_b200.impedances.impedance_sources import Resonators
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.trackers.tracker import RingAndRFTracker

pytestmark = pytest.mark.gpu


def _fused(n, S, precision, solver, **kw):
    turns = 24
    ring = Ring(6911.5, 1 / 18**2, 26e9, Proton(), turns)
    rf = RFStation(ring, [4620, 18480], [4.5e6, 4.5e5], [0.0, np.pi], n_rf=2)
    centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
    dt, dE = bigaussian_arrays(n, 0.4e-9, _get_dE_from_dt(ring, rf, 0.4e-9), centre, 5)
    beam = Beam(ring, n, 1e10, dt=dt, dE=dE, dtype=torch.float64)
    prof = Profile(beam, CutOptions(cut_left=centre - 1.25e-9, cut_right=centre + 1.25e-9,
                                    n_slices=S))
    iv = InducedVoltageFreq(beam, prof, [Resonators([2e5, 1e5], [200e6, 1.4e9],
                                                    [100.0, 3000.0])])
    return FusedTracker(RingAndRFTracker(rf, beam, solver=solver), prof,
                        TotalInducedVoltage(beam, prof, [iv]), precision=precision, **kw)


@pytest.mark.parametrize("n,precision,solver", [
    (5_000_001, "f64", "simple"), (2_000_000, "f64", "legacy"), (700_001, "f64", "exact"),
    (5_000_001, "q32p64", "simple"), (3_000_001, "f32p64", "exact")])
def test_same_bits_as_the_packed_pass(cuda, n, precision, solver):
    S = 65536
    tuned = _fused(n, S, precision, solver)
    choice = tuned.autotune()
    fixed = _fused(n, S, precision, solver, kernel="packed")
    for f in (tuned, fixed):
        f.track(4)
        f.check()
    assert torch.equal(tuned.dt, fixed.dt)
    assert torch.equal(tuned.dE, fixed.dE)
    assert torch.equal(tuned.profile_tensor(), fixed.profile_tensor())
    if choice["kernel"] != "packed" or choice["prefetch_stages"] != 1:
        pytest.skip(f"the autotuner picked {choice['kernel']}, ring "
                    f"{choice['prefetch_stages']}: other passes compared only")
