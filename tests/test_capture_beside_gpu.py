"""Calls on one stream while the caller captures another and forbids unsafe calls to
everyone (torch's default mode): uploads of pageable arrays keep the capture and
their own result, the first ever and later ones, on both sides of the largest size
that takes the page-locked stand-ins."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["pp", "bh"])
@pytest.mark.parametrize("n", [200, 16384, 16385])
@pytest.mark.parametrize("before", [0, 1, 2])
def test_upload_beside_a_capture(nb, cuda, mode, n, before):
    torch = cuda
    from nbody_gb300 import initializers as I

    systems = [nb.ParticleSystem(*I.uniform_ball(n, seed=s)) for s in (1, 2)]
    solver = nb.ParticleSolverCUDA(0.0035, 40.0, n, mode=mode)
    for _ in range(before):
        solver.upload(systems[0])
    captured, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    x = torch.zeros(4, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=captured, capture_error_mode="global"):
        x.add_(1)
        solver.upload(systems[0])
        solver.upload(systems[1])
        x.add_(1)
    graph.replay()
    torch.cuda.synchronize()
    assert x[0].item() == 2
    got = nb.ParticleSystem(np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32), np.zeros(n, np.float32))
    solver.download(got)
    np.testing.assert_array_equal(got.positions, systems[1].positions)
    np.testing.assert_array_equal(got.velocities, systems[1].velocities)
    solver.close()
