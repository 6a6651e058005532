"""Large host vectors through the handle's pinned buffers
(csrc/bdc_hostcopy.cu): the same values as through device memory, at sizes
around the threshold, with odd offsets and from several threads."""
import threading

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("n", [18, 20, 21, 23])
def test_host_vectors_round_trip(bdc, n):
    import torch
    with bdc.Engine(n, 3) as E:
        rng = np.random.default_rng(n)
        base = np.empty(E.R + 1, dtype=np.float64)
        for off in (0, 1):
            p = base[off:off + E.R]
            p[:] = rng.exponential(size=E.R)
            p /= 4.0 * p.sum()
            E.set_p(p)
            d = torch.empty(E.R, dtype=torch.float64, device="cuda")
            E.get_p_device(d.data_ptr())
            np.testing.assert_array_equal(d.cpu().numpy(), p)
            np.testing.assert_array_equal(E.get_p(), p)
            pinned = torch.from_numpy(p.copy()).pin_memory()
            out = torch.empty_like(pinned).pin_memory()
            E.baa_iteration_ptr(pinned.data_ptr(), out.data_ptr())
            np.testing.assert_array_equal(E.baa_iteration(p), out.numpy())


@pytest.mark.gpu
def test_handles_in_two_threads(bdc):
    res = {}

    def work(seed):
        with bdc.Engine(21, 4) as E:
            p = np.random.default_rng(seed).exponential(size=E.R)
            p /= 4.0 * p.sum()
            for _ in range(5):
                E.set_p(p)
                res.setdefault(seed, []).append(np.array_equal(E.get_p(), p))

    ts = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert res == {1: [True] * 5, 2: [True] * 5}


@pytest.mark.gpu
def test_fresh_and_resident_results(bdc):
    """A result of 33.6 MB into pages that are not there yet, at an odd offset,
    and into the same pages again."""
    import ctypes
    import mmap

    import torch
    with bdc.Engine(24, 3) as E:
        E.set_p(np.random.default_rng(4).exponential(size=E.R) / (4.0 * E.R))
        d = torch.empty(E.R, dtype=torch.float64, device="cuda")
        E.get_p_device(d.data_ptr())
        want = d.cpu().numpy()
        m = mmap.mmap(-1, 8 * E.R + 4096, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS)
        out = np.frombuffer(m, dtype=np.float64)[3:3 + E.R]
        for _ in range(2):
            assert bdc.library().bdc_get_p(E._h, out.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), E.R) == 0
            np.testing.assert_array_equal(out, want)
            out[:] = 0.0
