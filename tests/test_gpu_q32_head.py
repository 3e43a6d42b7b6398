"""Q32P64 turns keep the cluster FFT's roundings: the voltage of an engine and of
a batch equals, to the bit, the drop-in transform's of the same profile (which
takes that kernel below 2^13 complex points), and a beam tracked in a batch ends
on the same counts as one tracked alone."""
import pytest
import torch
from scipy.constants import e as E_CHARGE

from blond_b200 import bmath as bm
from blond_b200.batch import BatchTracker
from blond_b200.engine import FusedTracker
from blond_b200.trackers.tracker import RingAndRFTracker
from test_gpu_convolve import _objects

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [15, 177, 1000, 2048, 4096])
def test_voltage_is_the_cluster_transforms(cuda, S):
    rf, beam, prof, tiv = _objects(20001, S, S)
    iv = tiv.induced_voltage_list[0]
    one = FusedTracker(RingAndRFTracker(rf, beam), prof, tiv, precision="q32p64",
                       kernel="plain", energy_unit=1.0)
    many = BatchTracker([(RingAndRFTracker(r, b), p, t) for r, b, p, t in
                         (_objects(20001, S, S), _objects(3001, S, S + 1))],
                        precision="q32p64", energy_units=[1.0, 1.0])
    for _ in range(2):
        want = bm.induced_voltage_1turn(one.profile_tensor().clone(), iv.total_impedance,
                                        iv.n_fft, E_CHARGE * beam.ratio, S)
        one.track(1)
        many.track(1)
        assert torch.equal(one.induced_voltage_tensor(), want)
        assert torch.equal(many.induced_voltages_tensor()[0], want)
        assert torch.equal(many.dE[:20001], one.dE)
