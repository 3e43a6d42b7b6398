"""More beams in a batch than a grid has rows (65535), through the C ABI: the
impulse responses of short profiles are built for every one of them."""
import ctypes as ct

import numpy as np
import pytest
import torch

from blond_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S", [(65535, 4), (65536, 4), (70001, 8)])
def test_every_beam_has_its_voltage(cuda, B, S):
    turns, n_fft, per = 2, S + S % 2, 3
    rng = np.random.default_rng(B)
    ptr = lambda a: a.ctypes.data_as(ct.c_void_p)  # noqa: E731
    h = ct.c_void_p()
    call = lambda name, *a: _lib.call(f"blond_batch_{name}", h, *a)  # noqa: E731
    _lib.call("blond_batch_create", ct.byref(h), 0, B, 1, 0, S)
    try:
        prog = [np.full((B, turns + 1, 1), v) for v in (1e6, 1e9, 0.0)]
        acc = np.zeros((B, turns))
        call("set_rf", turns, *(ptr(a) for a in prog), ptr(acc), 1.0)
        drift = [np.full((B, turns + 1), v)
                 for v in (1e-6, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0, 1e9)]
        call("set_drift", 1.0, 0.0, *(ptr(a) for a in drift))
        cl, cr = np.zeros(B), np.full(B, 1e-9)
        bc = np.tile((np.arange(S) + 0.5) * (1e-9 / S), (B, 1))
        call("set_slicing", ptr(cl), ptr(cr), ptr(bc))
        Z = rng.normal(size=(B, n_fft // 2 + 1)) + 1j * rng.normal(size=(B, n_fft // 2 + 1))
        scale = rng.uniform(0.5, 2.0, B)
        call("set_impedance", n_fft, ptr(Z), ptr(scale))
        dt = torch.tensor(rng.uniform(0.0, 1e-9, B * per), device="cuda")
        dE = torch.zeros_like(dt)
        offsets = (per * np.arange(B + 1)).astype(np.int64)
        call("bind_beams", dt.data_ptr(), dE.data_ptr(), ptr(offsets))
        call("set_turn", 0, _lib.stream())
        call("slice", _lib.stream())
        p = torch.empty(B, S, dtype=torch.float64, device="cuda")
        v = torch.empty_like(p)
        call("get_profiles", p.data_ptr(), _lib.stream())
        call("run", 1, _lib.stream())
        call("get_induced_voltages", v.data_ptr(), _lib.stream())
        p, v = p.cpu().numpy(), v.cpu().numpy()
    finally:
        _lib.call("blond_batch_destroy", h)
    assert (p.sum(axis=1) == per).all()
    want = -scale[:, None] * np.fft.irfft(Z * np.fft.rfft(p, n_fft, axis=1), n_fft, axis=1)[:, :S]
    # at most 3 products of response and count, a response of at most 9 terms:
    # 20 roundings of sum |h| |p| <= 3 max |h|, and numpy's own
    bound = 40 * np.finfo(float).eps * 3 * scale * np.abs(Z).max(axis=1) * 2
    assert (np.abs(v - want) <= bound[:, None]).all()
