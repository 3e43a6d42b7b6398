"""Impedances put in one another's place on one engine, each of another kind of
head (convolution, 16-CTA power-of-two transform at n_fft or at a longer
length, mixed-radix transform): every turn has the voltage of the last one that
was accepted, as an engine that never had another gives it."""
import ctypes as ct

import numpy as np
import pytest
import torch

from blond_b200 import BlondB200Error
from blond_b200.batch import BatchTracker
from blond_b200.beam.beam import Beam, Proton
from blond_b200.beam.distributions import _get_dE_from_dt, bigaussian_arrays
from blond_b200.beam.profile import CutOptions, Profile
from blond_b200.engine import FusedTracker
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.trackers.tracker import RingAndRFTracker

pytestmark = pytest.mark.gpu


def _fused(S, precision, turns):
    ring = Ring(6911.5, 1 / 18**2, 26e9, Proton(), turns)
    rf = RFStation(ring, [4620], [4.5e6], [0.0])
    centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
    dt, dE = bigaussian_arrays(20001, 0.4e-9, _get_dE_from_dt(ring, rf, 0.4e-9), centre, S)
    beam = Beam(ring, len(dt), 1e10, dt=dt, dE=dE, dtype=torch.float64)
    prof = Profile(beam, CutOptions(cut_left=centre - 1.25e-9, cut_right=centre + 1.25e-9,
                                    n_slices=S))
    return FusedTracker(RingAndRFTracker(rf, beam), prof, precision=precision, kernel="plain",
                        energy_unit=1.0)


def _set(fused, n_fft, seed):
    rng = np.random.default_rng(seed)
    m = n_fft // 2 + 1
    Z = (rng.normal(size=m) + 1j * rng.normal(size=m)) / np.sqrt(m)
    fused.eng.call("set_impedance", n_fft, Z.ctypes.data_as(ct.c_void_p), 1.0 + seed)


@pytest.mark.parametrize("precision", ["f64", "f32p64", "q32p64"])
@pytest.mark.parametrize("S,lengths", [(600, [600, 8192, 648, 1024]),
                                       (5000, [5000, 8192, 16384, 6000]),
                                       (14000, [14400, 16384, 20000, 32768])])
def test_last_accepted_impedance(cuda, precision, S, lengths):
    one = _fused(S, precision, 2 * len(lengths) + 1)
    for k, n_fft in enumerate(lengths + lengths[::-1]):
        _set(one, n_fft, k)
        with pytest.raises(BlondB200Error):  # a factor of 7
            _set(one, 14 * S, 99)
        fresh = _fused(S, precision, 2 * len(lengths) + 1)
        fresh.dt.copy_(one.dt)
        fresh.dE.copy_(one.dE)
        fresh.eng.call("slice", torch.cuda.current_stream().cuda_stream)
        _set(fresh, n_fft, k)
        one.track(1)
        fresh.track(1)
        assert float(one.induced_voltage_tensor().abs().max()) > 0
        assert torch.equal(one.induced_voltage_tensor(), fresh.induced_voltage_tensor())
        assert torch.equal(one.dt, fresh.dt) and torch.equal(one.dE, fresh.dE)
    one.check()


@pytest.mark.parametrize("precision", ["f64", "q32p64"])
@pytest.mark.parametrize("B,S,lengths", [(3, 300, [300, 512, 324]), (40, 1200, [1200, 2048]),
                                         (2, 5000, [5000, 8192, 6000])])
def test_last_accepted_impedance_of_a_batch(cuda, precision, B, S, lengths):
    def build():
        items = []
        for b in range(B):
            ring = Ring(6911.5, 1 / 18**2, 26e9, Proton(), 2 * len(lengths))
            rf = RFStation(ring, [4620], [4.5e6], [0.0])
            centre = (rf.phi_s[0] - rf.phi_rf[0, 0]) / rf.omega_rf[0, 0]
            dt, dE = bigaussian_arrays(501 + b, 0.4e-9, 1e8, centre, b)
            beam = Beam(ring, len(dt), 1e10, dt=dt, dE=dE, dtype=torch.float64)
            items.append((RingAndRFTracker(rf, beam), Profile(beam, CutOptions(
                cut_left=centre - 1.25e-9, cut_right=centre + 1.25e-9, n_slices=S)), None))
        return BatchTracker(items, precision=precision, energy_units=[1.0] * B
                            if precision == "q32p64" else None)

    def put(batch, n_fft, seed):
        rng = np.random.default_rng(seed)
        m = n_fft // 2 + 1
        Z = (rng.normal(size=(B, m)) + 1j * rng.normal(size=(B, m))) / np.sqrt(m)
        scale = 1.0 + seed + np.arange(B)
        batch._call("set_impedance", n_fft, Z.ctypes.data_as(ct.c_void_p),
                    scale.ctypes.data_as(ct.c_void_p))

    one = build()
    for k, n_fft in enumerate(lengths + lengths[::-1]):
        put(one, n_fft, k)
        with pytest.raises(BlondB200Error):  # a factor of 7
            put(one, 14 * S, 99)
        fresh = build()
        fresh.dt.copy_(one.dt)
        fresh.dE.copy_(one.dE)
        fresh._call("slice", torch.cuda.current_stream().cuda_stream)
        put(fresh, n_fft, k)
        one.track(1)
        fresh.track(1)
        assert float(one.induced_voltages_tensor().abs().max()) > 0
        assert torch.equal(one.induced_voltages_tensor(), fresh.induced_voltages_tensor())
        assert torch.equal(one.dt, fresh.dt) and torch.equal(one.dE, fresh.dE)
    one.check()
