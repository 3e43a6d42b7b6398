"""The adjoint where the short-profile paths do not apply: more than 4600
slices at a power-of-two length transform once a turn (with the spectra
accumulated there and the deposit converted by the forward turn's last block),
more than 4266 gather the stored voltages from global memory while a segment is
recomputed, more than 14278 keep no block-private histogram.  70 turns in one
checkpoint interval: a segment of two launches.

Bars as in test_gpu_adjoint.py: coordinates within 1e-12 normwise of the numpy
restatement; a particle's weight in a bin then moves by at most 1e-12 max|dt| /
bin size and a bin holds at most about 2 max(p) particles, in either of two bins;
gradients within 1e-4 of central differences of the restatement.  Their relative
step, 3e-9, is on the plateau (differences at 1e-8 .. 1e-9 agree within 4e-5);
larger ones move particles across bin centres, where the map has kinks.  One
particle's own coordinates take 1e-7: their share of the loss is 1 / n.
"""
import numpy as np
import pytest
import torch

import adjoint_oracle as ao
from conftest import normwise
from test_gpu_adjoint import gpu_grads, make, oracle_args, oracle_loss

pytestmark = pytest.mark.gpu

RES = (np.array([1e6]), np.array([1e9]), np.array([1.0]))
T, STEP = 70, 3e-9


@pytest.mark.parametrize("S", [5000, 8192, 16384])
def test_forward_and_gradients(cuda, S):
    _, rf, tr, dt0, dE0, target = make(4000, S, T, K=T, intensity=3e9)
    x = dict(V=np.full((T, 1), 4.5e6), phi=np.zeros((T, 1)), R=RES[0], fr=RES[1], Q=RES[2],
             dt0=dt0, dE0=dE0)
    tg = target.cpu().numpy()
    L, g, (dt, dE, p) = gpu_grads(tr, dt0, dE0, x["V"], x["phi"], *RES, target)
    odt, odE, op, ov = ao.track(dt0, dE0, *oracle_args(tr, x["V"], x["phi"], *RES))
    assert normwise(dt.detach().cpu().numpy(), odt) < 1e-12
    assert normwise(dE.detach().cpu().numpy(), odE) < 1e-12
    assert normwise(p.detach().cpu().numpy(), op) < 4e-12 * np.abs(odt).max() * tr.inv_w
    assert np.abs(ov[-1]).max() > 1e3  # the induced voltage matters
    assert abs(L - oracle_loss(tr, dt0, dE0, x["V"], x["phi"], *RES, tg)) < 1e-11 * abs(L)
    for kind, idx, step in [("V", (0, 0), STEP), ("V", (T - 1, 0), STEP), ("R", 0, STEP),
                            ("Q", 0, STEP), ("dt0", 17, 1e-7), ("dE0", 17, 1e-7)]:
        h = step * (0.4e-9 if kind == "dt0" else abs(x[kind][idx]))
        f = []
        for s in (1, -1):
            a = {k: v.copy() for k, v in x.items()}
            a[kind][idx] += s * h
            f.append(oracle_loss(tr, a["dt0"], a["dE0"], a["V"], a["phi"], a["R"], a["fr"], a["Q"],
                                 tg))
        ref = (f[0] - f[1]) / (2 * h)
        rounding = 4 * np.finfo(float).eps * abs(L) / h
        assert abs(g[kind][idx] - ref) <= 1e-4 * abs(ref) + rounding, (kind, g[kind][idx], ref)


@pytest.mark.parametrize("S", [5000, 8192])
def test_checkpoint_interval_and_segments(cuda, S):
    out = []
    for K in (T, 64, 7):
        _, rf, tr, dt0, dE0, target = make(4000, S, T, K=K, intensity=3e9)
        out.append(gpu_grads(tr, dt0, dE0, np.full((T, 1), 4.5e6), np.zeros((T, 1)), *RES,
                             target)[1])
    for g in out[1:]:
        for k in g:
            assert normwise(g[k], out[0][k]) < 1e-12, k
