"""The reference's runs without collective effects, one turn a call: several
such turns in one call run in registers (particle_kernel_multi), so only single
ones go through the selected particle pass.  And the exact and legacy drift with
an impedance, where the pass and the graph of turns run: single turns against
graphs, and each kind of pass against the others, to the bit."""
import numpy as np
import pytest
import torch

from conftest import golden, normwise
from test_gpu_tracking import build, make_profile
from blond_b200.engine import FusedTracker
from blond_b200.impedances.impedance import InducedVoltageFreq, TotalInducedVoltage
from blond_b200.impedances.impedance_sources import Resonators
from blond_b200.trackers.tracker import RingAndRFTracker

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["track_rf.npz", "track_exact.npz", "track_legacy.npz"])
@pytest.mark.parametrize("kernel", ["tma", "plain"])
def test_reference_turn_by_turn(cuda, name, kernel):
    g = golden(name)
    ring, rf, beam = build(g)
    prof = make_profile(g, beam)
    fused = FusedTracker(RingAndRFTracker(rf, beam, solver=str(g["solver"][0])), prof, None,
                         precision="f64", kernel=kernel)
    nt = int(g["n_turns"][0])
    np.testing.assert_array_equal(fused.profile_tensor().cpu().numpy(), g["profiles"][0])
    for t in range(nt):
        fused.track(1)
        np.testing.assert_array_equal(fused.profile_tensor().cpu().numpy(), g["profiles"][t + 1])
    tol = 1e-10 if str(g["solver"][0]) != "simple" else 1e-11
    assert normwise(beam.dt.cpu().numpy(), g["dt"]) < tol
    assert normwise(beam.dE.cpu().numpy(), g["dE"]) < tol


@pytest.mark.parametrize("name", ["track_exact.npz", "track_legacy.npz"])
@pytest.mark.parametrize("precision", ["f64", "f32p64", "q32p64"])
def test_drifts_with_an_impedance(cuda, name, precision):
    g = golden(name)
    out = []
    for kernel, per_graph in (("plain", 3), ("plain", 1), ("tma", 3), ("packed", 3), ("stab", 3)):
        ring, rf, beam = build(g)
        prof = make_profile(g, beam)
        tiv = TotalInducedVoltage(beam, prof, [InducedVoltageFreq(
            beam, prof, [Resonators(5e6, 1e9, 1.0)])])
        fused = FusedTracker(RingAndRFTracker(rf, beam, solver=str(g["solver"][0])), prof, tiv,
                             precision=precision, kernel=kernel, turns_per_graph=per_graph,
                             energy_unit=1.0)
        fused.track(7)
        fused.check()
        assert float(fused.induced_voltage_tensor().abs().max()) > 0
        out.append((fused.dt.clone(), fused.dE.clone(), fused.profile_tensor(),
                    fused.induced_voltage_tensor()))
    for other in out[1:]:
        assert all(torch.equal(a, b) for a, b in zip(out[0], other))
