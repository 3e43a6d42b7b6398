"""The beam-phase loop inside the FFT head, which profiles too long for the
convolution and every Q32P64 engine take: power-of-two and padded lengths,
against the drop-in objects tracked turn by turn.

Bars: FP64 as in test_gpu_beam_feedback.py (trace and coordinates 1e-9, RF
programme 1e-12).  Q32P64, whose rounding of the energies this loop amplifies
from turn to turn, is checked turn by turn against the phase of its own profile:
S terms, each within 3 + |argument| roundings, added.
"""
import numpy as np
import pytest
import torch

from conftest import normwise
from blond_b200.beam.beam import Beam, Proton
from blond_b200.beam.distributions import bigaussian
from blond_b200.beam.profile import CutOptions, Profile
from blond_b200.engine import FusedTracker
from blond_b200.impedances.impedance import InducedVoltageFreq, TotalInducedVoltage
from blond_b200.impedances.impedance_sources import Resonators
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.llrf.beam_feedback import BeamFeedback
from blond_b200.trackers.tracker import FullRingAndRF, RingAndRFTracker

pytestmark = pytest.mark.gpu

TURNS = 50


def _objects(S, delay=0):
    ring = Ring(6911.5038, 1.0 / 17.95142852 ** 2, 25.92e9, Proton(), TURNS)
    rf = RFStation(ring, 4620, 4.5e6, 0)
    beam = Beam(ring, 200_000, 1e11)
    bigaussian(ring, rf, beam, 0.05e-9, seed=1234)
    beam.dt += 0.1e-9
    profile = Profile(beam, CutOptions(cut_left=0, cut_right=rf.t_rf[0, 0], n_slices=S))
    loop = BeamFeedback(ring, rf, profile, {"machine": "LHC_F", "PL_gain": 1000.0,
                                            "FL_gain": 0.05}, delay=delay)
    tracker = RingAndRFTracker(rf, beam, profile=profile, beam_feedback=loop)
    tiv = TotalInducedVoltage(beam, profile, [InducedVoltageFreq(
        beam, profile, [Resonators(5e6, 1e9, 1.0)])])
    return rf, beam, profile, loop, tracker, tiv


def _by_objects(S, delay):
    rf, beam, profile, loop, section, tiv = _objects(S, delay)
    tracker = FullRingAndRF([section])
    trace = np.zeros((TURNS, 3))
    for turn in range(TURNS):
        tiv.track()
        tracker.track()
        profile.track()
        trace[turn] = (loop.phi_beam, loop.dphi, loop.domega_rf)
    return rf, beam, trace


@pytest.mark.parametrize("S,delay", [(8192, 0), (8192, 7), (16384, 0), (14000, 0), (20000, 0)])
def test_loop_in_the_fft_head(cuda, S, delay):
    want_rf, want_beam, want = _by_objects(S, delay)
    rf, beam, profile, loop, tracker, tiv = _objects(S, delay)
    fused = FusedTracker(tracker, profile, tiv, precision="f64")
    fused.track(1)
    fused.track(TURNS - 1)
    fused.check()
    fused.sync()
    trace, x = fused.loop_trace[:TURNS], slice(delay, None)
    assert np.abs(want[x, 1]).max() > 0.01  # the loop has something to do
    for col in range(3):
        assert normwise(trace[x, col], want[x, col]) < 1e-9, col
    assert normwise(rf.omega_rf[0], want_rf.omega_rf[0]) < 1e-12
    assert normwise(rf.phi_rf[0], want_rf.phi_rf[0]) < 1e-9
    for a, b in ((beam.dt, want_beam.dt), (beam.dE, want_beam.dE)):
        assert normwise(a.cpu().numpy(), b.cpu().numpy()) < 1e-9


@pytest.mark.parametrize("S", [8, 1000, 1024, 8192])
@pytest.mark.parametrize("delay", [0, 3])
def test_q32p64_phase_of_its_profile(cuda, S, delay):
    rf, beam, profile, loop, tracker, tiv = _objects(S, delay)
    # (2.1 GeV of range: the shifted bunch and the strong resonator take it far)
    fused = FusedTracker(tracker, profile, tiv, precision="q32p64", energy_unit=1.0)
    bc = np.asarray(profile.bin_centers, float)
    w = np.ones(S)
    w[0] = w[-1] = 0.5
    for turn in range(8):
        p = fused.profile_tensor().cpu().numpy()
        x = rf.omega_rf[0, turn] * bc + rf.phi_rf[0, turn]
        fused.track(1)
        fused.check()
        fused.sync()
        if turn < delay:
            continue
        s, c = np.sum(w * p * np.sin(x)), np.sum(w * p * np.cos(x))
        bound = 2.0 ** -52 * (S + 10 + np.abs(x).max()) * p.sum() / np.hypot(s, c) + 2.0 ** -50
        assert abs(fused.loop_trace[turn][0] - (np.arctan(s / c) + np.pi)) <= bound
