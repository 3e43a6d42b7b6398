"""Host threads that call one bmath kernel with different profile lengths.

A kernel's dynamic shared memory limit belongs to the function, not to a
launch: were it set to each call's own need, a thread with a short profile
would lower it between another thread's setting and launch, and that launch
would be refused.  Every call has to succeed.  The threads call the entry
points by their bound functions, so that the calls come close together (the
interpreter lock is released inside them).
"""
import threading

import pytest
import torch

from blond_b200 import _lib

pytestmark = pytest.mark.gpu

# particles, profile lengths (one kernel each, some beyond the 48 KB a launch
# has without a raised limit; the interpolated kick's shared-memory table needs
# 400 particles per slice) and calls a thread
CASES = {"linear_interp_kick": (3_300_000, [8000, 100, 7000, 8], 20_000),
         "histogram": (2000, [20000, 9000, 15000, 8500], 60_000),
         "smooth_histogram": (2000, [20000, 100, 15000, 8], 60_000)}


@pytest.mark.parametrize("suffix", ["f64", "f32"])
@pytest.mark.parametrize("name", list(CASES))
def test_profile_lengths_of_other_threads(cuda, name, suffix):
    n, lengths, calls = CASES[name]
    dtype = torch.float64 if suffix == "f64" else torch.float32
    dt = torch.rand(n, device="cuda", dtype=dtype)
    fn = getattr(_lib.load(), f"blond_{name}_{suffix}")
    failures, keep, args = [], [], []
    for S in lengths:
        stream = torch.cuda.Stream()
        if name == "linear_interp_kick":
            t = [torch.zeros_like(dt), torch.rand(S, device="cuda", dtype=dtype),
                 torch.linspace(0.0, 1.0, S, device="cuda", dtype=dtype)]
            args.append((dt.data_ptr(), t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), 1.0,
                         S, n, 0.0, stream.cuda_stream))
        else:
            t = [torch.empty(S, device="cuda", dtype=dtype)]
            args.append((dt.data_ptr(), t[0].data_ptr(), 0.0, 1.0, S, n, stream.cuda_stream))
        keep.append((stream, t))
    torch.cuda.synchronize()
    start = threading.Barrier(len(lengths))

    def work(a):
        torch.cuda.set_device(0)
        start.wait()
        for _ in range(calls):
            rc = fn(*a)
            if rc:
                failures.append((a[4:], _lib.load().blond_b200_last_error().decode()))

    threads = [threading.Thread(target=work, args=(a,)) for a in args]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not failures, (len(failures), failures[0])
