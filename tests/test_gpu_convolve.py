"""The direct-convolution head against numpy's FFT on the same profile.

The head sums S products per output, as partial sums of at most 150 terms
and a tree over them; a response value carries the inverse FFT's error, a
few eps of its norm.  With |h| |p| summing to at most ~1e3 max|V| for these
resonators the bound is 200 eps x 1e3 = 4e-11 of max|V|.
"""
import numpy as np
import pytest
import torch
from scipy.constants import e as E_CHARGE

from conftest import normwise
from blond_b200.batch import BatchTracker
from blond_b200.beam.beam import Beam, Proton
from blond_b200.beam.distributions import _get_dE_from_dt, bigaussian_arrays
from blond_b200.beam.profile import CutOptions, Profile
from blond_b200.engine import FusedTracker
from blond_b200.impedances.impedance import (InducedVoltageFreq, InductiveImpedance,
                                             TotalInducedVoltage)
from blond_b200.impedances.impedance_sources import Resonators
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.trackers.tracker import RingAndRFTracker

pytestmark = pytest.mark.gpu
BAR = 4e-11


def _objects(n, S, seed, inductive=False, turns=4):
    ring = Ring(6911.5, 1 / 18**2, 26e9, Proton(), turns)
    rf = RFStation(ring, [4620], [4.5e6], [0.0])
    centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
    dt, dE = bigaussian_arrays(n, 0.4e-9, _get_dE_from_dt(ring, rf, 0.4e-9), centre, seed)
    beam = Beam(ring, n, 1e10, dt=dt, dE=dE, dtype=torch.float64)
    prof = Profile(beam, CutOptions(cut_left=centre - 1.25e-9, cut_right=centre + 1.25e-9,
                                    n_slices=S))
    parts = [InducedVoltageFreq(beam, prof, [Resonators([2e5, 1e5], [200e6, 1.4e9],
                                                        [100.0, 3000.0])])]
    if inductive:
        parts.append(InductiveImpedance(beam, prof, [0.01] * (turns + 1), rf))
    return rf, beam, prof, TotalInducedVoltage(beam, prof, parts)


def _voltage(p, rf, beam, prof, tiv, turn):
    iv = tiv.induced_voltage_list[0]
    v = -E_CHARGE * beam.ratio * np.fft.irfft(
        iv.total_impedance.cpu().numpy() * np.fft.rfft(p, iv.n_fft), iv.n_fft)[:len(p)]
    if len(tiv.induced_voltage_list) > 1:
        v = v - (E_CHARGE / (2 * np.pi) * beam.ratio * 0.01 * rf.t_rev[turn] / prof.bin_size
                 * np.gradient(p, prof.bin_centers[1] - prof.bin_centers[0]))
    return v


# tiles of 8 outputs less one per block: edges at 7, 8 and (8 g - 1) x 148;
# 4600 slices is the last profile of a power-of-two transform that convolves
@pytest.mark.parametrize("S", [4, 7, 8, 15, 201, 1036, 1037, 2220, 2221, 4096, 4600, 4601, 8192,
                               9000])
@pytest.mark.parametrize("form", ["f64", "f32p64", "inductive"])
def test_single_beam(cuda, S, form):
    rf, beam, prof, tiv = _objects(20001, S, S, inductive=form == "inductive")
    fused = FusedTracker(RingAndRFTracker(rf, beam), prof, tiv,
                         precision="f32p64" if form == "f32p64" else "f64", kernel="plain")
    for turn in range(2):
        p = fused.profile_tensor().cpu().numpy()
        assert p.sum() > 19000  # the histogram was cleared and refilled
        fused.track(1)
        want = _voltage(p, rf, beam, prof, tiv, turn)
        assert normwise(fused.induced_voltage_tensor().cpu().numpy(), want) < BAR
    assert fused.profile_tensor().sum() <= 20001
    fused.check()


@pytest.mark.parametrize("B,S", [(2, 7), (3, 300), (37, 400), (150, 64), (40, 1200)])
def test_batch(cuda, B, S):
    objs = [_objects(2000 + 7 * b, S, b) for b in range(B)]
    batch = BatchTracker([(RingAndRFTracker(rf, beam), prof, tiv)
                          for rf, beam, prof, tiv in objs], precision="f64")
    for turn in range(2):
        p = batch.profiles_tensor().cpu().numpy()
        batch.track(1)
        got = batch.induced_voltages_tensor().cpu().numpy()
        for b, (rf, beam, prof, tiv) in enumerate(objs):
            assert normwise(got[b], _voltage(p[b], rf, beam, prof, tiv, turn)) < BAR
