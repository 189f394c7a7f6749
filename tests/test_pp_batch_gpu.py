"""A system's last work item of the ensemble's direct sum runs with as many
bodies per thread as it needs: sizes on each side of every such count, against
the -v 2 port (ParticleSolverCPUParallel.cpp:27-40) under the direct-sum bounds
(per-body relative RMS <= 1e-5, max <= 1e-3), and the same bits from every
launch shape (the sum of a body runs over its system in one order in all)."""
import numpy as np
import pytest

from conftest import rel_err_stats

pytestmark = pytest.mark.gpu

SIZES = [2, 127, 128, 129, 255, 256, 257, 383, 384, 385, 511, 512, 513, 640, 641, 767, 768, 769, 895, 896, 897, 1025]


@pytest.mark.parametrize("eps2", [40.0, 0.0])
def test_last_items_of_every_length(nb, cuda, oracle, eps2):
    got = {}
    for shape in ("128x2", "256x2", "128x4", "256x4"):
        with nb.Ensemble(crossover=1 << 30, pp_shape=shape) as ens:
            ids = []
            for k, n in enumerate(SIZES):
                ids.append(ens.add(n, 0.0035, eps2))
                ens.init_device(ids[-1], "plummer", seed=300 + k, params=[50.0, 1.0, 20.0])
            start = [ens.download(i) for i in ids]
            ens.step(1)
            got[shape] = [ens.download(i) for i in ids]
    for k, n in enumerate(SIZES):
        out = got["128x4"][k]  # its accelerations are the forces at the step's start
        rms, mx = rel_err_stats(out.accelerations, oracle.pp_forces(start[k].positions, start[k].masses[:, 0], eps2))
        assert rms <= 1e-5 and mx <= 1e-3, (n, rms, mx)
        for shape in ("128x2", "256x2", "256x4"):
            np.testing.assert_array_equal(got[shape][k].positions, out.positions)
            np.testing.assert_array_equal(got[shape][k].velocities, out.velocities)
            np.testing.assert_array_equal(got[shape][k].accelerations, out.accelerations)
