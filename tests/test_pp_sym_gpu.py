"""The direct sum that evaluates every pair once (pp_sym.cu), against the -v 2
restatement (ParticleSolverCPUParallel.cpp:27-40) and the kernels over ordered
pairs, under the direct-sum bounds of tests/test_pp_gpu.py (per-body relative
RMS <= 1e-5, max <= 1e-3)."""
import numpy as np
import pytest

from conftest import rel_err_stats

pytestmark = pytest.mark.gpu


def _forces(nb, torch, solver, pm, n):
    f = torch.full((n, 4), float("nan"), dtype=torch.float32, device="cuda")
    solver.pp_forces_device(pm, f, n)
    solver.sync()
    return f.cpu().numpy()


def _solver(nb, torch, n, eps2):
    s = nb.ParticleSolverCUDA(0.0035, eps2, n, mode="pp")
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    return s


# One block and two (even and odd numbers of blocks), block and tile edges, a
# last block of one body, the smallest size that takes this path by itself, and
# softening zero.
@pytest.mark.parametrize("n,eps2", [(1, 40.0), (2, 0.0), (64, 40.0), (65, 40.0), (1023, 40.0), (1025, 0.0),
                                    (2048, 40.0), (3073, 40.0), (4096, 0.0), (10000, 40.0), (10241, 0.5),
                                    (15360, 40.0)])
def test_pp_sym_matches_port(nb, cuda, oracle, monkeypatch, n, eps2):
    torch = cuda
    from nbody_gb300 import initializers as I

    monkeypatch.setenv("NBODY_PP_SYM", "1")
    pos, _, mass = I.uniform_ball(n, seed=900 + n)
    pm = torch.from_numpy(I.pos_mass(pos, mass)).cuda()
    solver = _solver(nb, torch, n, eps2)
    assert solver.pp_config()["bodies_per_thread"] == 4
    got = _forces(nb, torch, solver, pm, n)
    np.testing.assert_array_equal(got, _forces(nb, torch, solver, pm, n))
    ref = oracle.pp_forces(pos, mass, eps2)
    assert np.all(got[:, 3] == 0)
    if n == 1:
        assert np.all(got == 0)
        return
    rms, mx = rel_err_stats(got, ref)
    assert rms <= 1e-5 and mx <= 1e-3, (rms, mx)


@pytest.mark.parametrize("scale,mass_scale,eps2", [(1e11, 1e6, 40.0), (1e-7, 1e-10, 1e-26), (1e10, 1.0, 1e30)])
def test_pp_sym_keeps_the_range_of_the_ordered_sum(nb, cuda, monkeypatch, scale, mass_scale, eps2):
    """Lengths whose inverse cube alone would leave FP32's range (1e-39 at 1e13,
    1e42 at 1e-14) and masses that bring the product back."""
    torch = cuda
    from nbody_gb300 import initializers as I

    n = 3000
    pos, _, mass = I.uniform_ball(n, seed=77)
    pm = torch.from_numpy(I.pos_mass(pos * np.float32(scale), mass * np.float32(mass_scale))).cuda()
    out = {}
    for sym in ("1", "0"):
        monkeypatch.setenv("NBODY_PP_SYM", sym)
        solver = _solver(nb, torch, n, eps2)
        out[sym] = _forces(nb, torch, solver, pm, n)
        solver.close()
    # relative, in units in which the squares do not underflow
    ref = out["0"].astype(np.float64)
    unit = np.abs(ref).max()
    assert np.isfinite(unit) and unit > 0
    rms, mx = rel_err_stats(out["1"] / unit, ref / unit)
    assert rms <= 1e-5 and mx <= 1e-3, (rms, mx)


def test_pp_sizes_alternate_on_one_context(nb, cuda):
    """One context serves bodies of several sizes in turn: each call gives what a
    fresh context gives, whatever its scratch held before."""
    torch = cuda
    from nbody_gb300 import initializers as I

    sizes = [131072, 5000, 12000, 16384, 5000, 131072, 2048, 12000]
    bodies = {n: torch.from_numpy(I.pos_mass(*(I.uniform_ball(n, seed=n)[k] for k in (0, 2)))).cuda() for n in set(sizes)}
    fresh = {}
    for n, pm in bodies.items():
        solver = _solver(nb, torch, n, 40.0)
        fresh[n] = _forces(nb, torch, solver, pm, n)
        solver.close()
    shared = _solver(nb, torch, 64, 40.0)
    for n in sizes:
        np.testing.assert_array_equal(_forces(nb, torch, shared, bodies[n], n), fresh[n])
