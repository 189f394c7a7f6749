"""The direct sum's launch shapes below 8,192 bodies (one or four bodies per
thread, short j-slices): each side of every change of shape against the -v 2
restatement (ParticleSolverCPUParallel.cpp:27-40), under the direct-sum bounds
(per-body relative RMS <= 1e-5, max <= 1e-3)."""
import numpy as np
import pytest

from conftest import rel_err_stats

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,eps2", [(31, 40.0), (32, 40.0), (95, 0.0), (96, 40.0), (128, 40.0), (129, 0.0), (1535, 40.0),
                                    (1536, 40.0), (3749, 40.0), (3750, 0.0), (6249, 40.0), (6250, 40.0), (6749, 0.0),
                                    (6750, 40.0), (8191, 40.0), (8192, 40.0)])
def test_pp_small_shapes_match_port(nb, cuda, oracle, n, eps2):
    from nbody_gb300 import initializers as I

    pos, vel, mass = I.uniform_ball(n, seed=500 + n)
    system = nb.ParticleSystem(pos.copy(), vel.copy(), mass)
    solver = nb.ParticleSolverCUDA(0.0035, eps2, n, mode="pp")
    solver.update_particle_positions(system)
    first = system.forces.copy()
    rms, mx = rel_err_stats(first, oracle.pp_forces(pos, mass, eps2))
    assert rms <= 1e-5 and mx <= 1e-3, (rms, mx)
    again = nb.ParticleSystem(pos.copy(), vel.copy(), mass)
    solver.update_particle_positions(again)
    np.testing.assert_array_equal(again.forces, first)
    np.testing.assert_array_equal(again.positions, system.positions)
    solver.close()
