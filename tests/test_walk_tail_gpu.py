"""The last sets of a large system, walked by larger teams in a launch beside the
others': each side of both changes of size, odd numbers of bodies, against one
warp per set throughout. A body meets exactly the records of its own reference
walk either way (src/Octree/Octree.cpp:303-338), so the counted pairs are equal;
the sums are taken in another order (the direct-sum bounds: per-body relative
RMS <= 1e-5, max <= 1e-3), and a system has the same bits alone, through host
arrays and in an ensemble."""
import numpy as np
import pytest

from conftest import rel_err_stats
from test_walk_team_gpu import _forces

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,eps2", [(131072, 40.0), (131073, 40.0), (131200, 0.0), (262143, 10.0), (458752, 40.0),
                                    (458753, 0.0), (600001, 40.0)])
def test_tail_walk_matches_one_warp_per_set(nb, cuda, monkeypatch, n, eps2):
    torch = cuda
    from nbody_gb300 import initializers as I

    pos, _, mass = I.plummer(n, a=100.0, seed=n % 1000)
    pm = torch.from_numpy(I.pos_mass(pos, mass)).cuda()
    got, pairs = _forces(nb, torch, pm, n, 0.25, eps2)
    monkeypatch.setenv("NBODY_BH_TEAM", "1")
    ref, ref_pairs = _forces(nb, torch, pm, n, 0.25, eps2)
    assert pairs == ref_pairs
    rms, mx = rel_err_stats(got, ref)
    assert rms <= 1e-5 and mx <= 1e-3, (rms, mx)


def test_tail_walk_system_is_the_same_alone_on_host_arrays_and_in_an_ensemble(nb, cuda):
    sizes = [131073, 470001, 5000, 40000]
    with nb.Ensemble(crossover=0) as ens:
        ids = [ens.add(n, 0.0035, 40.0, 0.25, mode="bh") for n in sizes]
        for k, sid in enumerate(ids):
            ens.init_device(sid, "plummer", seed=70 + k)
        start = [ens.download(sid) for sid in ids]
        ens.step(2, graph_steps=2)
        got = [ens.download(sid) for sid in ids]
    for k, n in enumerate(sizes):
        for host in (False, True):
            one = nb.ParticleSolverCUDA(0.0035, 40.0, n, mode="bh", theta2=0.25)
            z = np.zeros((n, 4), np.float32)
            ref = nb.ParticleSystem(z, z.copy(), np.zeros(n, np.float32))
            if host:
                ref = nb.ParticleSystem(start[k].positions.copy(), start[k].velocities.copy(), start[k].masses.copy(),
                                        start[k].accelerations.copy())
                for _ in range(2):
                    one.update_particle_positions(ref)
            else:
                one.init_device("plummer", seed=70 + k)
                one.step(2)
                one.download(ref)
            one.close()
            np.testing.assert_array_equal(got[k].positions, ref.positions)
            np.testing.assert_array_equal(got[k].velocities, ref.velocities)
            np.testing.assert_array_equal(got[k].accelerations, ref.accelerations)
