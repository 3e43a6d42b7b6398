"""Prefetch 1, which the autotuner reports for the packed pass's register
pipeline, can be set like the other depths: the packed pass's bits with it, and
direct loads in the passes that have no such pipeline."""
import numpy as np
import pytest
import torch

from blond_b200 import BlondB200Error
from blond_b200.beam.beam import Beam, Proton
from blond_b200.beam.distributions import _get_dE_from_dt, bigaussian_arrays
from blond_b200.beam.profile import CutOptions, OtherSlicesOptions, Profile
from blond_b200.engine import FusedTracker
from blond_b200.impedances.impedance import InducedVoltageFreq, TotalInducedVoltage
from blond_b200.impedances.impedance_sources import Resonators
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.trackers.tracker import RingAndRFTracker

pytestmark = pytest.mark.gpu


def _run(n, S, precision, solver, kernel, prefetch, interpolation=False, smooth=False, imp=True):
    turns = 6
    ring = Ring(6911.5, 1 / 18**2, 26e9, Proton(), turns)
    rf = RFStation(ring, [4620, 18480], [4.5e6, 4.5e5], [0.0, np.pi], n_rf=2)
    centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
    dt, dE = bigaussian_arrays(n, 0.4e-9, 1e8, centre, n)
    dt[::97] += 2e-9  # some particles beyond the window
    beam = Beam(ring, n, 1e10, dt=dt, dE=dE, dtype=torch.float64)
    prof = Profile(beam, CutOptions(cut_left=centre - 1.25e-9, cut_right=centre + 1.25e-9,
                                    n_slices=S),
                   other_slices_options=OtherSlicesOptions(smooth=smooth))
    tiv = None
    if imp:
        tiv = TotalInducedVoltage(beam, prof, [InducedVoltageFreq(
            beam, prof, [Resonators([2e5, 1e5], [200e6, 1.4e9], [100.0, 3000.0])])])
    fused = FusedTracker(RingAndRFTracker(rf, beam, solver=solver, interpolation=interpolation,
                                          profile=prof if interpolation else None,
                                          total_induced_voltage=tiv if interpolation else None),
                         prof, tiv, precision=precision, kernel=kernel, energy_unit=1.0)
    fused.eng.call("set_prefetch", prefetch)
    fused.track(3)
    fused.check()
    return fused.dt, fused.dE, fused.profile_tensor()


def _same(a, b):
    assert all(torch.equal(x, y) for x, y in zip(a, b))
    assert torch.isfinite(a[0]).all()


# 148 blocks x 768 threads: a thread has no pair, one, two and three (227328,
# 454656, 681984 particles are the edges), and the odd particle
@pytest.mark.parametrize("n", [1, 2, 1537, 227_329, 454_656, 681_985, 900_001])
@pytest.mark.parametrize("precision", ["f64", "f32p64", "q32p64"])
@pytest.mark.parametrize("solver", ["simple", "legacy", "exact"])
def test_pipeline_same_bits_as_the_packed_pass(cuda, n, precision, solver):
    _same(_run(n, 4096, precision, solver, "packed", 1),
          _run(n, 4096, precision, solver, "packed", 0))


@pytest.mark.parametrize("precision", ["f64", "f32p64", "q32p64"])
@pytest.mark.parametrize("S,interpolation", [(4, False), (1000, True), (65536, False),
                                             (65536, True)])
def test_pipeline_profile_lengths_and_interpolated_kick(cuda, precision, S, interpolation):
    _same(_run(300_001, S, precision, "simple", "packed", 1, interpolation),
          _run(300_001, S, precision, "simple", "packed", 0, interpolation))


# 57000 slices leave no room for a ring stage beside the histogram
@pytest.mark.parametrize("S,kernel,smooth,imp", [
    (1000, "plain", False, True), (1000, "tma", False, True), (1000, "stab", False, True),
    (57000, "plain", False, False), (1000, "plain", True, True)])
def test_other_passes_take_direct_loads(cuda, S, kernel, smooth, imp):
    _same(_run(50_001, S, "f64", "simple", kernel, 1, smooth=smooth, imp=imp),
          _run(50_001, S, "f64", "simple", kernel, 0, smooth=smooth, imp=imp))


def test_other_depths_are_refused(cuda):
    for bad in (-1, 3, 5):
        with pytest.raises(BlondB200Error):
            _run(10, 10, "f64", "simple", "plain", bad)
