"""The 16-CTA power-of-two transform (head_fft.cu) against torch's FFT.

Two transforms of M = N / 2 points lose about eps log2(M) each against the
largest output: 2 x 15 x 1.1e-16 and the products' roundings, bar 1e-14 of
max|V|.  The table it writes is checked through the kick it gives: the same
turn with the table gathered (plain pass) and with the entries formed from the
voltages (shared-table pass) has to give the same bits.
"""
import numpy as np
import pytest
import torch
from scipy.constants import e as E_CHARGE

from conftest import normwise
from blond_b200 import bmath as bm
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
BAR = 1e-14


@pytest.mark.parametrize("N", [8192, 16384, 32768, 65536, 131072])
def test_induced_voltage(cuda, N):
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    for S, n_out in ((N, N), (N - 1, N - 1), (N // 2 + 3, N), (1, 5), (N, 1)):
        p = torch.randn(S, generator=g, device="cuda", dtype=torch.float64)
        Z = torch.view_as_complex(torch.randn(N // 2 + 1, 2, generator=g, device="cuda",
                                              dtype=torch.float64))
        v = bm.induced_voltage_1turn(p, Z, N, 2.0, n_out)
        want = -2.0 * torch.fft.irfft(Z * torch.fft.rfft(p, N), N)
        assert float((v - want[:n_out]).abs().max() / want.abs().max()) < BAR, S


def _run(S, kernel, precision, inductive):
    turns = 3
    ring = Ring(6911.5, 1 / 18**2, 26e9, Proton(), turns)
    rf = RFStation(ring, [4620], [4.5e6], [0.0])
    centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
    dt, dE = bigaussian_arrays(100001, 0.4e-9, _get_dE_from_dt(ring, rf, 0.4e-9), centre, S)
    beam = Beam(ring, len(dt), 1e10, dt=dt, dE=dE, dtype=torch.float64)
    prof = Profile(beam, CutOptions(cut_left=centre - 1.25e-9, cut_right=centre + 1.25e-9,
                                    n_slices=S))
    parts = [InducedVoltageFreq(beam, prof, [Resonators([2e5, 1e5], [200e6, 1.4e9],
                                                        [100.0, 3000.0])])]
    if inductive:
        parts.append(InductiveImpedance(beam, prof, [1e-4] * (turns + 1), rf))
    tiv = TotalInducedVoltage(beam, prof, parts)
    fused = FusedTracker(RingAndRFTracker(rf, beam), prof, tiv, precision=precision,
                         kernel=kernel)
    for t in range(2):
        p = fused.profile_tensor().cpu().numpy()
        assert p.sum() > 99000  # cleared and refilled
        fused.track(1)
        iv = parts[0]
        want = -E_CHARGE * beam.ratio * np.fft.irfft(
            iv.total_impedance.cpu().numpy() * np.fft.rfft(p, iv.n_fft), iv.n_fft)[:S]
        if inductive:
            want = want - (E_CHARGE / (2 * np.pi) * beam.ratio * 1e-4 * rf.t_rev[t]
                           / prof.bin_size * np.gradient(p, prof.bin_centers[1]
                                                         - prof.bin_centers[0]))
        assert normwise(fused.induced_voltage_tensor().cpu().numpy(), want) < BAR
    fused.check()
    return fused.dt, fused.dE


# from 9325 slices on no convolution takes the profile; other lengths than a
# power of two go through one of at least twice the profile
@pytest.mark.parametrize("S", [8192, 9600, 16384, 20000, 32768, 40000, 49152, 65536])
@pytest.mark.parametrize("form", ["f64", "f32p64", "inductive"])
def test_engine_head(cuda, S, form):
    precision = "f32p64" if form == "f32p64" else "f64"
    got = _run(S, "plain", precision, form == "inductive")
    if S <= 16384:  # within the shared table's limit
        other = _run(S, "stab", precision, form == "inductive")
        assert torch.equal(got[0], other[0]) and torch.equal(got[1], other[1])
