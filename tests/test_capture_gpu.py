"""Calls made while the caller captures the context's stream, replayed later: the
direct sum at sizes whose plans lay out the scratch differently, each replay
between the others' (and eager calls between them), and an upload of pageable
arrays, which a replay reads as they are then."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_captured_direct_sums_replay_between_each_other(nb, cuda):
    torch = cuda
    from nbody_gb300 import initializers as I

    sizes = [300, 5003, 8200, 12000, 20011, 40000]
    stream = torch.cuda.Stream()
    solver = nb.ParticleSolverCUDA(0.0035, 40.0, max(sizes), mode="pp")
    solver.set_stream(stream.cuda_stream)
    pm, out, want, graphs = {}, {}, {}, {}
    with torch.cuda.stream(stream):
        for n in sizes:
            pos, _, mass = I.uniform_ball(n, seed=n)
            pm[n] = torch.from_numpy(I.pos_mass(pos, mass)).cuda()
            out[n] = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        for n in reversed(sizes):  # the largest scratch first: it does not move afterwards
            solver.pp_forces_device(pm[n], out[n], n)
            solver.sync()
            want[n] = out[n].clone()
    torch.cuda.synchronize()
    for n in sizes:
        graphs[n] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs[n], stream=stream, capture_error_mode="thread_local"):
            solver.pp_forces_device(pm[n], out[n], n)
    rng = np.random.default_rng(1)
    with torch.cuda.stream(stream):
        for n in [int(x) for x in rng.choice(sizes, 24)]:
            out[n].fill_(float("nan"))
            if rng.random() < 0.3:
                solver.pp_forces_device(pm[n], out[n], n)
            else:
                graphs[n].replay()
            solver.sync()
            assert torch.equal(out[n], want[n]), n
    solver.close()


@pytest.mark.parametrize("mode", ["pp", "bh"])
def test_captured_upload_reads_the_arrays_at_replay(nb, cuda, mode):
    torch = cuda
    from nbody_gb300 import initializers as I

    n = 777
    pos, vel, mass = I.uniform_ball(n, seed=3)
    stream = torch.cuda.Stream()
    solver = nb.ParticleSolverCUDA(0.0035, 40.0, n, mode=mode)
    solver.set_stream(stream.cuda_stream)
    system = nb.ParticleSystem(pos.copy(), vel.copy(), mass.copy(), np.zeros_like(pos))
    solver.upload(system)
    solver.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        solver.upload(system)
    system.positions[:, :3] *= 2.0
    system.velocities[:, :3] += 1.0
    with torch.cuda.stream(stream):
        graph.replay()
    got = nb.ParticleSystem(np.zeros_like(pos), np.zeros_like(pos), np.zeros_like(mass))
    solver.download(got)
    np.testing.assert_array_equal(got.positions, system.positions)
    np.testing.assert_array_equal(got.velocities, system.velocities)
    solver.close()
