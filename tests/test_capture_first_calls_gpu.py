"""The first direct sum of a context made while the caller captures its stream: small
sums need no allocation then (up to 510 bodies), and give the bits of an eager call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["pp", "bh"])
@pytest.mark.parametrize("n", [1, 95, 96, 200, 256, 480, 510])
def test_first_call_under_capture(nb, cuda, mode, n):
    torch = cuda
    from nbody_gb300 import initializers as I

    pos, _, mass = I.uniform_ball(n, seed=n)
    pm = torch.from_numpy(I.pos_mass(pos, mass)).cuda()
    want, got = torch.zeros((n, 4), device="cuda"), torch.full((n, 4), float("nan"), device="cuda")
    eager = nb.ParticleSolverCUDA(0.0035, 40.0, n, mode=mode)
    eager.pp_forces_device(pm, want, n)
    eager.sync()
    eager.close()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    solver = nb.ParticleSolverCUDA(0.0035, 40.0, n, mode=mode)
    solver.set_stream(stream.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="global"):
        solver.pp_forces_device(pm, got, n)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    solver.sync()
    np.testing.assert_array_equal(got.cpu().numpy(), want.cpu().numpy())
    solver.close()
