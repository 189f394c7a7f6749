"""The cell walk by teams of warps (walk_team.cu) against the one-warp cell
walk and the union walk.

All forms give a body exactly the records its own reference walk accepts
(src/Octree/Octree.cpp:303-338), so the counted pair evaluations are equal;
the sums are taken in another order, which in FP32 moves a force by the
rounding of some 10^3 .. 10^4 terms: the direct-sum bounds of the other tests
(per-body relative RMS <= 1e-5, max <= 1e-3).
"""
import numpy as np
import pytest

from conftest import rel_err_stats

pytestmark = pytest.mark.gpu

# (bodies, theta^2, eps^2): partial and single sets, both sides of every
# change of team size, a small opening angle (more open cells than a team's
# stack holds, so subtrees go to the union walk), and eps^2 = 0.
CASES = [(1, 0.25, 40.0), (2, 0.25, 40.0), (63, 0.25, 40.0), (65, 0.25, 40.0), (129, 0.25, 0.0), (5000, 0.01, 40.0),
         (10239, 0.25, 40.0), (10240, 0.25, 40.0), (20000, 0.01, 40.0), (32767, 0.36, 10.0), (32768, 0.25, 0.0),
         (40000, 0.01, 40.0)]


def _forces(nb, torch, pm, n, theta2, eps2):
    solver = nb.ParticleSolverCUDA(0.0035, eps2, n, mode="bh", theta2=theta2)
    solver.set_stream(torch.cuda.current_stream().cuda_stream)
    out = []
    for count in (False, False, True):
        if count:
            solver.bh_counters(True)
        f = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        solver.bh_forces_device(pm, f)
        solver.sync()
        out.append(f.cpu().numpy())
    pairs = solver.bh_counters(False)[0]
    solver.close()
    np.testing.assert_array_equal(out[0], out[1])  # the same bits on every run
    return out[0], pairs


@pytest.mark.parametrize("n,theta2,eps2", CASES)
def test_team_walk_matches_the_other_forms(nb, cuda, monkeypatch, n, theta2, eps2):
    torch = cuda
    from nbody_gb300 import initializers as I

    pos, _, mass = I.plummer(n, a=100.0, seed=100 + n)
    pm = torch.from_numpy(I.pos_mass(pos, mass)).cuda()
    got, pairs = _forces(nb, torch, pm, n, theta2, eps2)
    forms = {"team1": ("NBODY_BH_TEAM", "1"), "team2": ("NBODY_BH_TEAM", "2"), "team4": ("NBODY_BH_TEAM", "4"),
             "team8": ("NBODY_BH_TEAM", "8"), "team16": ("NBODY_BH_TEAM", "16"), "union": ("NBODY_BH_WALK", "union")}
    for name, (var, value) in forms.items():
        monkeypatch.setenv(var, value)
        ref, ref_pairs = _forces(nb, torch, pm, n, theta2, eps2)
        monkeypatch.delenv(var)
        assert pairs == ref_pairs, name
        if n > 1:
            rms, mx = rel_err_stats(got, ref)
            assert rms <= 1e-5 and mx <= 1e-3, (name, rms, mx)


def test_team_walk_system_is_the_same_alone_and_in_an_ensemble(nb, cuda):
    """Systems of every team size in one ensemble: each the single solver's bits."""
    sizes = [600, 10240, 20000, 33000, 10239]
    with nb.Ensemble(crossover=0) as ens:
        ids = [ens.add(n, 0.0035, 40.0, 0.25, mode="bh") for n in sizes]
        for k, sid in enumerate(ids):
            ens.init_device(sid, "plummer", seed=50 + k)
        ens.step(3, graph_steps=2)
        got = [ens.download(sid) for sid in ids]
    for k, n in enumerate(sizes):
        one = nb.ParticleSolverCUDA(0.0035, 40.0, n, mode="bh", theta2=0.25)
        one.init_device("plummer", seed=50 + k)
        one.step(3)
        z = np.zeros((n, 4), np.float32)
        ref = nb.ParticleSystem(z, z.copy(), np.zeros(n, np.float32))
        one.download(ref)
        one.close()
        np.testing.assert_array_equal(got[k].positions, ref.positions)
        np.testing.assert_array_equal(got[k].velocities, ref.velocities)
        np.testing.assert_array_equal(got[k].accelerations, ref.accelerations)
