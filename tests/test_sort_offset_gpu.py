"""nbody_sort_pairs_device on slices that begin anywhere a key and a value may, not
at a multiple of 16 bytes: both sides of the sizes at which the sort changes its
form (2,048 and 2^18 pairs, 2^22 + 1), against numpy's stable argsort."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [None, "merge", "radix"])
@pytest.mark.parametrize("n", [2049, 262144, 262145, 300001, 4194305])
def test_sort_of_slices(nb, cuda, monkeypatch, form, n):
    torch = cuda
    if form:
        monkeypatch.setenv("NBODY_SORT", form)
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 40, n, dtype=np.uint64)
    keys[rng.random(n) < 0.3] = np.uint64(7)
    vals = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    order = np.argsort(keys, kind="stable")
    solver = nb.ParticleSolverCUDA(0.0035, 40.0, 64, mode="bh")
    solver.set_stream(torch.cuda.current_stream().cuda_stream)
    for ko, vo in [(1, 0), (0, 1), (1, 3), (0, 2)]:
        kbuf = torch.full((n + 4,), -1, dtype=torch.int64, device="cuda")
        vbuf = torch.full((n + 4,), -1, dtype=torch.int32, device="cuda")
        k, v = kbuf[ko:ko + n], vbuf[vo:vo + n]
        k.copy_(torch.from_numpy(keys.view(np.int64)))
        v.copy_(torch.from_numpy(vals.view(np.int32)))
        rc = nb.lib().nbody_sort_pairs_device(solver._ctx, ctypes.c_void_p(k.data_ptr()),
                                              ctypes.c_void_p(v.data_ptr()), n)
        assert rc == nb.OK
        solver.sync()
        np.testing.assert_array_equal(k.cpu().numpy().view(np.uint64), keys[order])
        np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), vals[order])
        for buf, at in ((kbuf, ko), (vbuf, vo)):  # nothing written beside the slice
            assert int((buf[:at] != -1).sum()) == 0 and int((buf[at + n:] != -1).sum()) == 0
    solver.close()
