"""The bmath kernels on both sides of the sizes where they change their
launch: 1212416 particles (four a thread on 148 SMs), twice that for the
kick, 400 particles per slice for the interpolated kick's shared tables.

Histogram counts are exact (the same two rounded operations per particle).
The kick's increment carries the sine's 2 units in the last place and three
roundings: 1e-15 x (largest increment) in float64, 1e-6 in float32.  The
interpolated kick is compared in the reference's own form, whose terms
t slope and bc slope cancel: each operation rounds once, 4 eps max|bc slope|.
"""
import numpy as np
import pytest
import torch

from blond_b200 import bmath as bm

pytestmark = pytest.mark.gpu
SIZES = [1, 31, 300001, 1212415, 1212416, 2424833, 6553600, 6553601]


def _beam(n, dtype):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    dt = torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * 0.5e-9 + 2.5e-9
    dE = torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * 2e7
    dt[n // 2] = float("nan")
    return dt.to(dtype), dE.to(dtype)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", SIZES)
def test_histogram_counts(cuda, n, dtype):
    dt, _ = _beam(n, dtype)
    cl, cr = np.array([1.25e-9, 3.75e-9], np.float64 if dtype == torch.float64 else np.float32)
    for S in (1, 30, 2048, 8192, 8193, 30001):
        out = torch.full((S,), 7.0, dtype=dtype, device="cuda")
        bm.slice_beam(dt, out, float(cl), float(cr))
        inv_w = float(cl.dtype.type(S) / (cr - cl))
        f = torch.floor((dt - float(cl)) * inv_w)
        k = f[(f >= 0) & (f < S)].long()
        assert torch.equal(out, torch.bincount(k, minlength=S).to(dtype)), S


@pytest.mark.parametrize("dtype,bar", [(torch.float64, 1e-15), (torch.float32, 1e-6)])
@pytest.mark.parametrize("n", SIZES)
def test_kick(cuda, n, dtype, bar):
    for V, om, ph in (([4.5e6], [1.26e9], [0.1]), ([4.5e6, 4e5], [1.26e9, 5.04e9], [0.1, 3.0])):
        dt, dE = _beam(n, dtype)
        p = [torch.tensor(x, dtype=dtype, device="cuda") for x in (V, om, ph)]
        arg = [(p[1][j].double() * dt.double() + p[2][j].double()) for j in range(len(V))]
        if dtype == torch.float32:  # the kernel's argument in its own precision
            arg = [torch.addcmul(p[2][j].expand_as(dt), p[1][j], dt).double()
                   for j in range(len(V))]
        want = dE.double() + sum(p[0][j].double() * torch.sin(arg[j])
                                 for j in range(len(V))) - 1e3
        bm.kick(dt, dE, *p, 1.0, len(V), -1e3)
        err = (dE.double() - want).abs().nan_to_num(0.0).max()
        # one rounding of dE (1e8) beside the increment's own error
        assert float(err) <= bar * 5e6 + 1.2e8 * torch.finfo(dtype).eps
        assert int(torch.isnan(dE).sum()) == 1


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", SIZES)
def test_interpolated_kick(cuda, n, dtype):
    for S in (2, 1000, 16384, 29000):
        dt, dE = _beam(n, dtype)
        bc = torch.linspace(1.25e-9, 3.75e-9, S, dtype=torch.float64, device="cuda").to(dtype)
        v = (1e5 * torch.sin(torch.arange(S, device="cuda", dtype=torch.float64) * 0.01)).to(dtype)
        before = dE.clone()
        bm.linear_interp_kick(dt, dE, v, bc, 1.0, 0.0)
        inv_w = (S - 1) / (bc[-1] - bc[0])
        f = torch.floor((dt - bc[0]) * inv_w)
        inside = (f >= 0) & (f < S - 1)
        k = f.nan_to_num(0.0).clamp(0, S - 2).long()
        slope = (v[k + 1].double() - v[k].double()) * inv_w.double()
        offset = v[k].double() - bc[k].double() * slope
        want = torch.where(inside, before.double() + (dt.double() * slope + offset),
                           before.double())
        eps = torch.finfo(dtype).eps
        bar = 4 * eps * (float((bc[k].double() * slope).abs().max()) + 1.2e8)
        err = (dE.double() - want).abs().nan_to_num(0.0).max()
        assert float(err) <= bar, S
        # outside the table the energy stays as it is
        assert torch.equal(dE[~inside], before[~inside])
