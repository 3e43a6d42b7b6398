"""The particle pass with its own smooth deposit: the profile it leaves equals,
to the bit, the one blond_engine_slice takes of the same coordinates (64-bit
sums), and without induced voltage the coordinates equal those of the turn with
integer slicing.  28000 slices still fit its shared memory, 30000 do not."""
import pytest
import torch

from blond_b200.beam.profile import OtherSlicesOptions, Profile
from blond_b200.engine import FusedTracker, _stream
from blond_b200.trackers.tracker import RingAndRFTracker
from test_gpu_multi_turn import _fused

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f64", "f32p64", "q32p64"])
@pytest.mark.parametrize("n,S,solver,n_rf", [
    (1, 2, "simple", 1), (2, 10, "legacy", 1), (2047, 100, "exact", 2), (100003, 600, "simple", 3),
    (400001, 1000, "exact", 1), (303105, 28000, "simple", 2), (60001, 30000, "legacy", 1)])
def test_profile_is_the_separate_deposit(cuda, precision, n, S, solver, n_rf):
    plain = _fused(n, S, 4, precision, solver, n_rf)
    f = _fused(n, S, 4, precision, solver, n_rf)
    smooth = Profile(f.beam, f.profile.cut_options,
                     other_slices_options=OtherSlicesOptions(smooth=True))
    f = FusedTracker(RingAndRFTracker(f.rf, f.beam, solver=solver), smooth, precision=precision,
                     kernel="plain", energy_unit=1.0, turns_per_graph=2)
    for turns in (1, 2):
        f.track(turns)
        plain.track(turns)
        got = f.profile_tensor().clone()
        f.eng.call("slice", _stream())
        assert torch.equal(got, f.profile_tensor())
        assert torch.equal(f.dt, plain.dt)
        assert torch.equal(f.dE, plain.dE)
