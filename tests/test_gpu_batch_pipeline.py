"""The batched pass's full iterations (loads of the next one in flight, no
lane tests) against its general form (the one that aggregated deposits take),
and the F32P64 slice index taken by a rounded-down addition.

A particle's arithmetic is the same in both forms, so coordinates and counts
are equal to the bit; beam sizes around a full iteration of 256 threads with
2, 4 and 8 particles a thread, odd starts included.
"""
import numpy as np
import pytest
import torch

from blond_b200.batch import BatchTracker
from blond_b200.trackers.tracker import RingAndRFTracker
from test_gpu_batch import make_beam

pytestmark = pytest.mark.gpu

TURNS = 3


def tracked(counts, precision, shape):
    built = [make_beam(k, n, TURNS) for k, n in enumerate(counts)]
    batch = BatchTracker([(RingAndRFTracker(rf, beam), prof, tiv)
                          for _, rf, beam, prof, tiv, _, _ in built], precision=precision,
                         energy_units=[0.5] * len(counts) if precision == "q32p64" else None)
    batch.set_shape(*shape)
    batch.track(TURNS)
    batch.check()
    return batch.dt.cpu(), batch.dE.cpu(), batch.profiles_tensor().cpu()


@pytest.mark.parametrize("precision", ["f64", "f32p64", "q32p64"])
@pytest.mark.parametrize("ppt", [2, 4, 8])
def test_full_iterations_are_the_general_form(cuda, precision, ppt):
    tile = 256 * ppt
    counts = [1, 63, 65, tile - 1, tile, tile + 1, 2 * tile - 2, 2 * tile, 2 * tile + 3,
              3 * tile - 63, 5 * tile + 64, 5 * tile + 1]
    want = tracked(counts, precision, (256, 1, 2, 4096, True))
    for chunk in (1 << 14, 3 * tile + 1):
        got = tracked(counts, precision, (256, 1, ppt, chunk, False))
        for g, w in zip(got, want):
            assert torch.equal(g, w)


def test_f32p64_slice_index_at_edges_and_outside(cuda):
    """Initial slicing against floor((dt - cut_left) / width) in doubles: slice
    edges and their neighbours, the window's ends, far outside, infinities."""
    ring, rf, beam, prof, tiv, _, _ = make_beam(0, 4096, TURNS)
    S, cl = prof.n_slices, float(prof.cut_left)
    edges = np.linspace(cl, float(prof.cut_right), S + 1)
    dt = np.concatenate([edges, np.nextafter(edges, -np.inf), np.nextafter(edges, np.inf),
                         [cl - 1.0, -1e300, 1e300, np.inf, -np.inf, np.nan, 1e9, -1e9, 0.0,
                          cl + 2.0**31 * (edges[1] - cl), cl + 2.0**32 * (edges[1] - cl),
                          cl + (2.0**32 + 3) * (edges[1] - cl)]])
    dt = np.concatenate([dt, np.full(4096 - len(dt), -1.0)])
    beam.dt.copy_(torch.as_tensor(dt))
    batch = BatchTracker([(RingAndRFTracker(rf, beam), prof, tiv)], precision="f32p64")
    got = batch.profiles_tensor().cpu().numpy()[0]
    inv_w = S / (float(prof.cut_right) - cl)
    y = (dt - cl) * inv_w
    ok = (y >= 0) & (y < S)
    want = np.bincount(np.floor(y[ok]).astype(int), minlength=S)
    np.testing.assert_array_equal(got, want)
