"""blond_induced_voltage_f32 against the float64 entry on the same profile: the
transform is the same, so its rounded result is equal to the bit.  Lengths on the
two transform kernels (below and from 2^13 complex points), a non-power of two,
profiles shorter and longer than the transform."""
import numpy as np
import pytest
import torch

from blond_b200 import bmath as bm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_fft,S,n_out", [(2, 1, 1), (1000, 1000, 1000), (1024, 700, 700),
                                           (1024, 1500, 1024), (4050, 2000, 0),
                                           (16384, 10001, 10001), (65536, 65536, 65535)])
def test_same_transform(cuda, n_fft, S, n_out):
    rng = np.random.default_rng(n_fft + S)
    p = torch.as_tensor(rng.integers(0, 1000, S).astype(np.float32), device="cuda")
    Z = torch.as_tensor(rng.normal(size=n_fft // 2 + 1) + 1j * rng.normal(size=n_fft // 2 + 1),
                        device="cuda")
    want = bm.induced_voltage_1turn(p.double(), Z, n_fft, 1.6e-9, n_out)
    got = bm.induced_voltage_1turn(p, Z, n_fft, 1.6e-9, n_out, torch.float32)
    assert want.dtype == torch.float64 and got.dtype == torch.float32
    assert torch.equal(got, want.float())
    # a float32 profile without a type keeps the float64 result
    assert torch.equal(bm.induced_voltage_1turn(p, Z, n_fft, 1.6e-9, n_out), want)
