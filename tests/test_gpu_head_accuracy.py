"""The heads' voltages against the same transform in extended precision, at the
edges of the convolution's tiles and of its range, in each of its forms.

Bars, u = 2^-53.  Convolution: a voltage is a sum of S products in partial sums
of at most seg terms, a tree over 32 wpg of them and a scale, (seg + 10 + wpg) u
sum |h| p; its responses are an inverse FFT of N values, 5 u log2(N) in the
2-norm, which through p is at most that |h|_2 |p|_2.  The padded power-of-two
transform (a response by an inverse and a forward transform, then two more):
four times eps log2(M) <= 4 x 15 x 1.1e-16 and the products, 2e-14 of max|V|.
"""
import numpy as np
import pytest
import torch
from scipy.constants import e as E_CHARGE

from blond_b200.beam.beam import Beam, Proton
from blond_b200.beam.distributions import bigaussian_arrays
from blond_b200.beam.profile import CutOptions, OtherSlicesOptions, Profile
from blond_b200.engine import FusedTracker
from blond_b200.impedances.impedance import InducedVoltageFreq, TotalInducedVoltage
from blond_b200.impedances.impedance_sources import Resonators
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.llrf.beam_feedback import BeamFeedback
from blond_b200.trackers.tracker import RingAndRFTracker

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
SOURCES = {"usual": ([2e5, 1e5], [200e6, 1.4e9], [100.0, 3000.0]),
           # 50 ps period and a long ring: a smooth bunch's products cancel
           "cancelling": ([1e6], [20e9], [1e4])}


def _fused(S, form="plain", source="usual", precision="f64", kernel="plain", turns=4):
    ring = Ring(6911.5, 1 / 18**2, 26e9, Proton(), turns)
    rf = RFStation(ring, [4620], [4.5e6], [0.0])
    centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
    dt, dE = bigaussian_arrays(20001, 0.4e-9, 1e8, centre, S)
    beam = Beam(ring, len(dt), 1e10, dt=dt, dE=dE, dtype=torch.float64)
    prof = Profile(beam, CutOptions(cut_left=centre - 1.25e-9, cut_right=centre + 1.25e-9,
                                    n_slices=S),
                   other_slices_options=OtherSlicesOptions(smooth=form == "smooth"))
    iv = InducedVoltageFreq(beam, prof, [Resonators(*SOURCES[source])])
    tiv = TotalInducedVoltage(beam, prof, [iv])
    loop = BeamFeedback(ring, rf, prof, {"machine": "LHC_F", "PL_gain": 1000.0,
                                         "FL_gain": 0.05}) if form == "loop" else None
    interp = form == "interpolated"
    tracker = RingAndRFTracker(rf, beam, profile=prof, beam_feedback=loop, interpolation=interp,
                               total_induced_voltage=tiv if interp else None)
    return FusedTracker(tracker, prof, tiv, precision=precision, kernel=kernel), iv, rf, prof


def _exact(p, iv, scale):
    """(voltage, sum |h| p per output, |h|_2): extended precision."""
    n, S = iv.n_fft, len(p)
    Z = iv.total_impedance.cpu().numpy().astype(np.clongdouble)
    pl = np.zeros(n, np.longdouble)
    pl[:S] = p
    v = -scale * np.fft.irfft(Z * np.fft.rfft(pl), n)[:S]
    h = np.fft.irfft(Z, n)
    both = np.fft.irfft(np.fft.rfft(np.abs(h)) * np.fft.rfft(pl), n)[:S]
    return v, scale * both, scale * np.sqrt(np.sum(h * h))


def _conv_bound(p, iv, scale):
    S, sms = len(p), torch.cuda.get_device_properties(0).multi_processor_count
    g = next(g for g in range(1, 13) if (8 * g - 1) * sms >= S)
    wpg = 4 if g <= 4 else (2 if g <= 8 else 1)
    seg = -(-S // (32 * wpg)) | 1
    _, both, h2 = _exact(p, iv, scale)
    return (seg + 10 + wpg) * U * both + 5 * U * np.log2(iv.n_fft) * h2 * np.sqrt(np.sum(p * p))


EDGES = [4, 7, 8, 1036, 1037, 2220, 2221, 4600]  # tiles of 8 outputs less one, 148 SMs
# no power of two: two warps and one a tile, and the last profile that fits
LONG = [5000, 9324, 9325, 12000, 13920]


@pytest.mark.parametrize("form,source", [("plain", "usual"), ("plain", "cancelling"),
                                         ("smooth", "usual"), ("interpolated", "usual"),
                                         ("loop", "usual")])
@pytest.mark.parametrize("S", EDGES + LONG)
def test_convolution(cuda, S, form, source):
    fused, iv, rf, prof = _fused(S, form, source)
    scale = E_CHARGE * fused.beam.ratio * 1.0
    for _ in range(2):
        p = fused.profile_tensor().cpu().numpy()
        fused.track(1)
        want = _exact(p, iv, scale)[0]
        got = fused.induced_voltage_tensor().cpu().numpy()
        assert (np.abs(got - want) <= _conv_bound(p, iv, scale)).all()
    fused.check()


@pytest.mark.parametrize("S", [13921, 14000, 15000, 16000])
@pytest.mark.parametrize("form", ["plain", "smooth", "interpolated", "loop"])
def test_long_profile_of_another_length(cuda, S, form):
    """From 13921 slices on, a power of two of at least twice the profile."""
    fused, iv, rf, prof = _fused(S, form)
    scale = E_CHARGE * fused.beam.ratio
    for _ in range(2):
        p = fused.profile_tensor().cpu().numpy()
        fused.track(1)
        want = _exact(p, iv, scale)[0]
        got = fused.induced_voltage_tensor().cpu().numpy()
        assert np.abs(got - want).max() <= 2e-14 * np.abs(want).max()
    fused.check()


@pytest.mark.parametrize("S", EDGES + LONG + [8192, 14000])
def test_loop_phase(cuda, S):
    """The beam phase of a turn from its profile, trapezoid sums over all
    slices: each term within 3 + |argument| roundings, S of them added."""
    fused, iv, rf, prof = _fused(S, "loop")
    p = fused.profile_tensor().cpu().numpy()
    bc = np.asarray(prof.bin_centers, float)
    fused.track(1)
    fused.sync()
    x = rf.omega_rf[0, 0] * bc + rf.phi_rf[0, 0]
    w = np.ones(S)
    w[0] = w[-1] = 0.5
    s, c = np.sum(w * p * np.sin(x)), np.sum(w * p * np.cos(x))
    bound = 2 * U * (S + 10 + np.abs(x).max()) * p.sum() / np.hypot(s, c) + 8 * U
    assert abs(fused.loop_trace[0][0] - (np.arctan(s / c) + np.pi)) <= bound


@pytest.mark.parametrize("S", EDGES + LONG + [8192, 14000])
def test_interpolated_kick(cuda, S):
    """RF and induced voltage from the head's table: the kick of a turn against
    the interpolation of the same voltages, each product of it rounded."""
    fused, iv, rf, prof = _fused(S, "interpolated")
    t, e0 = (a.cpu().numpy().copy() for a in (fused.dt, fused.dE))
    fused.track(1)
    v = fused.induced_voltage_tensor().cpu().numpy()
    bc = np.asarray(prof.bin_centers, float)
    arg = rf.omega_rf[0, 0] * bc + rf.phi_rf[0, 0]
    v = v + rf.voltage[0, 0] * np.sin(arg)
    v_err = U * ((np.abs(arg).max() + 4) * rf.voltage[0, 0] + np.abs(v).max())
    inv_w = (S - 1) / (bc[-1] - bc[0])
    f = np.floor((t - bc[0]) * inv_w)
    inside = (f >= 0) & (f < S - 1)
    k = f[inside].astype(int)
    slope = (v[k + 1] - v[k]) * inv_w
    want = e0.copy()
    want[inside] += (t[inside] - bc[k]) * slope + v[k]
    bound = np.full(len(t), 2 * U) * np.abs(e0)
    bound[inside] += 8 * U * (np.abs(t[inside] * slope) + np.abs(bc[k] * slope)
                              + np.abs(v[k])) + 4 * v_err
    assert inside.sum() > 15000
    assert (np.abs(fused.dE.cpu().numpy() - want) <= bound).all()
