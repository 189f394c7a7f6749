"""Pageable uploads of a small system on one stream, then on another: the second
upload's arrays must not reach what the first, still waiting on its own stream,
has yet to read."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WAIT_CYCLES = 200_000_000  # about 0.1 s of a bounded device-side wait in front of the first upload


class _View:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n, 4), "typestr": "<f4", "data": (int(ptr), False), "version": 3}


@pytest.mark.parametrize("mode", ["pp", "bh"])
@pytest.mark.parametrize("between", ["sync", "nothing", "close"])
def test_upload_on_another_stream_leaves_the_first_one_alone(nb, cuda, mode, between):
    torch = cuda
    from nbody_gb300 import initializers as I

    n = 3001
    systems = []
    for seed in (1, 2):
        pos, vel, mass = I.uniform_ball(n, seed=seed)
        systems.append(nb.ParticleSystem(pos, vel, mass))
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    solver = nb.ParticleSolverCUDA(0.0035, 40.0, n, mode=mode)
    solver.upload(systems[1])  # the stand-ins are made, the state is the second system's
    solver.sync()
    solver.set_stream(first.cuda_stream)
    with torch.cuda.stream(first):
        torch.cuda._sleep(WAIT_CYCLES)
        solver.upload(systems[0])
        state = torch.as_tensor(_View(solver.device_state()[0], n), device="cuda").clone()
    if between == "close":
        solver.close()
    else:
        solver.set_stream(second.cuda_stream)
        if between == "sync":
            solver.sync()
        second.wait_stream(first)
        solver.upload(systems[1])
        got = nb.ParticleSystem(np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32), np.zeros(n, np.float32))
        solver.download(got)
        np.testing.assert_array_equal(got.positions, systems[1].positions)
        np.testing.assert_array_equal(got.velocities, systems[1].velocities)
        solver.close()
    first.synchronize()
    np.testing.assert_array_equal(state.cpu().numpy()[:, :3], systems[0].positions[:, :3])
