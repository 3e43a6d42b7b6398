"""RingAndRFTracker's host side, without a GPU: which call the kick takes, and
the RF phase accumulation."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from blond_b200 import bmath as bm
from blond_b200.beam.beam import Proton
from blond_b200.input_parameters.rf_parameters import RFStation
from blond_b200.input_parameters.ring import Ring
from blond_b200.trackers.tracker import RingAndRFTracker


def _tracker(n_turns=4, n_rf=2):
    ring = Ring(6911.5, 1 / 18**2, 26e9, Proton(), n_turns)
    rf = RFStation(ring, [4620, 18480][:n_rf], [4.5e6, 4.5e5][:n_rf], [0.0, np.pi][:n_rf],
                   n_rf=n_rf)
    beam = SimpleNamespace(dt=torch.zeros(8, dtype=torch.float64),
                           dE=torch.zeros(8, dtype=torch.float64), particle=Proton())
    return rf, RingAndRFTracker(rf, beam)


# (device, dtype) of the coordinates; the programme's copy is float64 on the CPU
@pytest.mark.parametrize("device,dtype,direct", [("cpu", torch.float64, True),
                                                 ("cpu", torch.float32, False),
                                                 ("meta", torch.float64, False)])
@pytest.mark.parametrize("index", [0, 3, -1])
def test_kick_passes_addresses_only_to_arrays_beside_them(monkeypatch, device, dtype, direct,
                                                          index):
    rf, tracker = _tracker()
    V, om, ph = tracker._programme()
    calls = []
    monkeypatch.setattr(bm, "_check_particles", lambda *a: None)
    monkeypatch.setattr(bm, "_kick", lambda *a: calls.append(("address", a)))
    monkeypatch.setattr(bm, "kick", lambda *a: calls.append(("row", a)))
    dt = torch.zeros(8, dtype=dtype, device=device)
    tracker.kick(dt, torch.zeros_like(dt), index)
    (kind, a), = calls
    if direct and index >= 0:
        assert kind == "address"
        assert a[2:5] == (V[index].data_ptr(), om[index].data_ptr(), ph[index].data_ptr())
    else:
        assert kind == "row"
        assert all(torch.equal(x, y[index]) for x, y in zip(a[2:5], (V, om, ph)))


def _phase_after_a_turn(dphi_rf, offset, monkeypatch):
    """phi_rf of the next turn and dphi_rf after one turn that starts with
    ``dphi_rf`` and has the frequency ``offset`` beside the design one."""
    rf, tracker = _tracker()
    rf.empty = True  # no kick
    monkeypatch.setattr(bm, "drift", lambda *a: None)
    rf.omega_rf[:, 1] += np.asarray(offset)
    rf.dphi_rf = dphi_rf
    tracker.track()
    return rf.phi_rf[:, 1], rf.dphi_rf


@pytest.mark.parametrize("dphi", [np.zeros(2), np.array([0.25, -0.5]), 0.25, np.float64(0.5),
                                  np.array([0.5, 0.25], np.float32),
                                  np.array([0.5, np.nan])],
                         ids=["zeros", "values", "float", "scalar", "float32", "nan"])
@pytest.mark.parametrize("offset", [[0.0, 0.0], [1e3, -2e3]], ids=["design", "offset"])
def test_phase_offset_of_every_kind(monkeypatch, dphi, offset):
    """The frequency offset's phase is added to dphi_rf, as an array expression
    over the RF systems adds it, and the sum to the next turn's phase."""
    rf, _ = _tracker()
    od, h = rf.omega_rf_d[:, 1], rf.harmonic[:, 1]
    om = rf.omega_rf[:, 1] + np.asarray(offset)
    want = dphi.copy() if isinstance(dphi, np.ndarray) else dphi
    want += 2.0 * np.pi * h * (om - od) / od
    phi, got = _phase_after_a_turn(dphi, offset, monkeypatch)
    np.testing.assert_array_equal(got, want)
    assert np.asarray(got).dtype == np.asarray(want).dtype
    np.testing.assert_array_equal(phi, rf.phi_rf[:, 1] + want)


def test_phase_offset_of_whole_numbers_is_refused(monkeypatch):
    """Fractions of a radian cannot be added to an integer array in place."""
    with pytest.raises(TypeError):
        _phase_after_a_turn(np.zeros(2, int), [1e3, 0.0], monkeypatch)
