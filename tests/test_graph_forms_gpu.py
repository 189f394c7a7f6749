"""A context that has captured its step takes another kernel form from the next call
on: the bits of the same calls launched kernel by kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(nb, torch, monkeypatch, mode, n, var, values, graphs):
    from nbody_gb300 import initializers as I

    pin = lambda a: torch.from_numpy(a.copy()).pin_memory().numpy()  # noqa: E731
    pos, vel, mass = I.plummer(n, a=100.0, seed=n)
    monkeypatch.setenv("NBODY_GRAPHS", graphs)
    solver = nb.ParticleSolverCUDA(0.0035, 40.0, n, mode=mode)
    system = nb.ParticleSystem(pos, vel, mass)
    for name in ("positions", "velocities", "accelerations", "masses", "forces"):
        setattr(system, name, pin(getattr(system, name)))
    out, resident = [], []
    for value in values:
        if value is None:
            monkeypatch.delenv(var, raising=False)
        else:
            monkeypatch.setenv(var, value)
        if mode == "bh":  # resident steps, one graph per parity, and a host call
            solver.upload(system)
            solver.step(4)
            solver.download(system)
            resident = [system.positions.copy(), system.accelerations.copy()]
        solver.update_particle_positions(system)
        out.append(resident + [system.positions.copy(), system.accelerations.copy()])
    monkeypatch.delenv(var, raising=False)
    solver.close()
    return out


@pytest.mark.parametrize("mode,n,var,values", [
    ("bh", 5000, "NBODY_BH_TEAM", [None, "1", "4", None]),
    ("bh", 140000, "NBODY_BH_TEAM", [None, "1", None]),
    ("bh", 5000, "NBODY_SORT", [None, "radix", "merge"]),
    ("bh", 5000, "NBODY_UPSWEEP", [None, "levels", "climb"]),
    ("pp", 12000, "NBODY_PP_SYM", [None, "0", "1", None]),
    ("pp", 3000, "NBODY_PP_SLICES", [None, "3", None]),
])
def test_form_changed_after_a_capture(nb, cuda, monkeypatch, mode, n, var, values):
    replayed = _run(nb, cuda, monkeypatch, mode, n, var, values, "1")
    direct = _run(nb, cuda, monkeypatch, mode, n, var, values, "0")
    for got, want in zip(replayed, direct):
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)


def test_ensemble_form_changed_after_a_capture(nb, cuda, monkeypatch):
    """The sort's and the upsweep's forms give the same bits, replayed or not."""
    got = []
    for graph_steps in (2, 0):
        with nb.Ensemble(crossover=0) as ens:
            for k, n in enumerate([600, 3000]):
                ens.init_device(ens.add(n, 0.0035, 40.0, 0.25, mode="bh"), "plummer", seed=k)
            for var, value in [(None, None), ("NBODY_SORT", "radix"), ("NBODY_UPSWEEP", "climb")]:
                if var:
                    monkeypatch.setenv(var, value)
                ens.step(4, graph_steps=graph_steps)
                if var:
                    monkeypatch.delenv(var)
            got.append([ens.download(s).accelerations for s in (0, 1)])
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
