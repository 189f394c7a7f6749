"""Host calls on pageable arrays, which small systems take through page-locked
stand-ins: the bits of the same calls on page-locked arrays, on both sides of
the largest size that does, also with arrays that are not 16-byte aligned and
with arrays reused right after the upload."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _unaligned(a):
    buf = np.empty(a.nbytes + 4, np.uint8)
    view = buf[4:].view(np.float32).reshape(a.shape)
    view[:] = a
    return view


@pytest.mark.parametrize("mode", ["pp", "bh"])
@pytest.mark.parametrize("n,steps", [(1, 1), (2, 0), (777, 1), (777, 3), (16384, 1), (16385, 1)])
def test_pageable_calls_match_page_locked(nb, cuda, mode, n, steps):
    torch = cuda
    from nbody_gb300 import initializers as I

    pos, vel, mass = I.uniform_ball(n, seed=n)
    mass4 = np.zeros((n, 4), np.float32)
    mass4[:, 0] = mass
    start = [pos, vel, np.zeros_like(pos), mass4, np.zeros_like(pos)]
    pin = lambda a: torch.from_numpy(a.copy()).pin_memory().numpy()  # noqa: E731
    forms = {"locked": [pin(a) for a in start], "pageable": [a.copy() for a in start],
             "unaligned": [_unaligned(a) for a in start]}
    L = nb.lib()
    for name, arrays in forms.items():
        solver = nb.ParticleSolverCUDA(0.0035, 40.0, n, mode=mode)
        for _ in range(2):
            rc = L.nbody_update_host(solver._ctx, *[ctypes.c_void_p(a.ctypes.data) for a in arrays], steps)
            assert rc == nb.OK
        # upload, the arrays overwritten at once, step, download
        copies = [a.copy() for a in arrays] if name != "locked" else [pin(a) for a in arrays]
        rc = L.nbody_upload(solver._ctx, *[ctypes.c_void_p(a.ctypes.data) for a in copies[:4]])
        assert rc == nb.OK
        if name == "locked":
            solver.sync()
        for a in copies:
            a[:] = np.nan
        solver.step(1)
        rc = L.nbody_download(solver._ctx, *[ctypes.c_void_p(copies[k].ctypes.data) for k in (0, 1, 2, 4)])
        assert rc == nb.OK
        forms[name] = arrays + [copies[k] for k in (0, 1, 2, 4)]
        solver.close()
    for name in ("pageable", "unaligned"):
        for got, want in zip(forms[name], forms["locked"]):
            np.testing.assert_array_equal(got, want)
