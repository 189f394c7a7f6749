"""Workloads this library is timed on, through its public entry points.

Every case is one of four uses of the library, at sizes its command line, tests, benchmark and serving loop use:

  host      update_particle_positions on host arrays: the drop-in call of the reference's solver interface, one time
            step per call, arrays pageable (plain numpy) or page-locked
  steps     a run from a given state: upload, several steps in HBM, the state read back
  forces    accelerations of bodies already on the device, for a caller with its own integrator
  ensemble  many independent systems of uneven size stepped together and read back

for the direct sum ("pp") and Barnes-Hut ("bh"). Bodies come from the three synthetic shapes the library's workloads
use: a uniform ball (masses 1 .. 10, at rest), an equal-mass Plummer sphere in equilibrium, and two exponential discs
with a heavy centre each.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "n-body_gb300"))

import nbody_gb300 as nb  # noqa: E402

BASE = {"dt": 0.0035, "eps2": 40.0, "theta2": 0.25, "keys": "octree", "integrator": "cpu", "pinned": True}
# What the ensemble autotuner's stored result for this GPU says.
CROSSOVER, PP_SHAPE = 10050, "128x4"


def _case(name, use, solver, shape, n, **more):
    return {"name": name, "use": use, "solver": solver, "shape": shape, "n": n, **BASE, **more}


def listed():
    return [
        # The reference's own scale for a CPU run (its fixtures hold 1,000 bodies), from plain numpy arrays: latency.
        _case("pp_host_1000", "host", "pp", "ball", 1000, pinned=False),
        # The direct-sum benchmark: one drop-in call per step on page-locked arrays, and the same system kept resident.
        _case("pp_host_16384", "host", "pp", "ball", 16384),
        _case("pp_steps_16384", "steps", "pp", "ball", 16384, steps=20),
        # Device-resident callers: an odd middle size, and the largest direct sum in ordinary use.
        _case("pp_forces_5003", "forces", "pp", "plummer", 5003, eps2=10.0),
        _case("pp_forces_131071", "forces", "pp", "ball", 131071),
        # Barnes-Hut from the smallest systems it is meant for, as a first user calls it.
        _case("bh_host_4096", "host", "bh", "plummer", 4096, pinned=False),
        # A ragged middle size with the wider opening angle and the GLSL path's key.
        _case("bh_forces_30001", "forces", "bh", "ball", 30001, theta2=0.36, keys="morton"),
        # A resident run of a quarter of a million bodies with the GLSL path's integrator.
        _case("bh_steps_262144", "steps", "bh", "plummer", 262144, steps=10, integrator="gpu_euler"),
        # The Barnes-Hut benchmark: 2^20 bodies, one drop-in call per step on page-locked arrays.
        _case("bh_host_1048576", "host", "bh", "plummer", 1048576),
        # The scale workload: two discs of 2^23 bodies.
        _case("bh_forces_16777216", "forces", "bh", "discs", 16777216, theta2=0.36),
        # Ensembles: many small systems (all direct sum), and the ragged mix of the batched workload.
        _case("ens_512_small", "ensemble", "auto", "plummer", 512, lo=256, hi=4096, steps=10),
        _case("ens_128_ragged", "ensemble", "auto", "plummer", 128, lo=256, hi=131072, steps=10),
    ]


def _log_int(rng, lo, hi):
    return int(min(hi, math.floor(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    # eps2 0.0935 is the command line's default softening, 10 .. 40 what the serving loop's requests carry
    use = rng.choice(["host", "host", "steps", "steps", "forces", "forces", "ensemble"])
    c = {"use": use, **BASE, "dt": rng.choice([0.001, 0.0035]), 
         "eps2": rng.choice([0.0935, round(rng.uniform(10.0, 40.0), 3), round(rng.uniform(10.0, 40.0), 3)]),
         "theta2": rng.choice([0.25, 0.25, 0.36]), "keys": rng.choice(["octree", "octree", "morton"]),
         "integrator": rng.choice(["cpu", "cpu", "gpu_euler"]), "pinned": rng.random() < 0.6}
    if use == "ensemble":
        hi = rng.choice([4096, 16384, 131072])
        c.update(solver="auto", shape="plummer", n=_log_int(rng, 16, 512 if hi == 4096 else 100), lo=256, hi=hi,
                 steps=rng.choice([1, 5, 10]))
        return c
    c["solver"] = rng.choice(["pp", "bh"])
    if c["solver"] == "pp":
        c["shape"] = rng.choice(["ball", "plummer"])
        c["n"] = _log_int(rng, 256, 131071)
    else:
        c["shape"] = rng.choice(["plummer", "discs"] if use == "host" else ["ball", "plummer", "discs"])
        c["n"] = _log_int(rng, 2048, 1048576 if use == "steps" else 4194304)
    if c["shape"] == "discs":
        c["n"] += c["n"] % 2
    if use == "steps":
        c["steps"] = rng.choice([2, 5, 10]) if c["n"] > 32768 else rng.choice([5, 10, 20])
    return c


# ------------------------------------------------------------------ inputs
def _unit(n, g):
    d = torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
    return d / d.norm(dim=1, keepdim=True)


def _uniform(n, g):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _ball(n, g, radius=100.0):
    pos = radius * _uniform(n, g).pow(1.0 / 3.0)[:, None] * _unit(n, g)
    return pos, torch.zeros_like(pos), 1.0 + 9.0 * _uniform(n, g)


def _plummer(sizes, g, a=100.0):
    """Equal-mass Plummer spheres of scale a, one after the other."""
    # radii by inverse transform, truncated at 20 a; speeds q = v / v_esc from q^2 (1 - q^2)^3.5 by rejection
    n = sum(sizes)
    total = torch.repeat_interleave(torch.tensor(sizes, device="cuda"), torch.tensor(sizes, device="cuda")).double()
    top = 20.0**3 / (20.0**2 + 1.0) ** 1.5
    u = (_uniform(n, g) * top).clamp_min(1e-12)
    r = a / torch.sqrt(u.pow(-2.0 / 3.0) - 1.0)
    q = torch.zeros(n, device="cuda", dtype=torch.float64)
    todo = torch.arange(n, device="cuda")
    while todo.numel():
        x, y = _uniform(todo.numel(), g), 0.1 * _uniform(todo.numel(), g)
        ok = y < x * x * (1.0 - x * x).pow(3.5)
        q[todo[ok]] = x[ok]
        todo = todo[~ok]
    v_esc = torch.sqrt(2.0 * total / torch.sqrt(r * r + a * a))
    return r[:, None] * _unit(n, g), (q * v_esc)[:, None] * _unit(n, g), torch.ones_like(r)


def _discs(n, g, scale=200.0, height=20.0, centre=1e6, apart=2000.0, speed=50.0, tilt=30.0):
    halves = []
    for side in (-0.5, 0.5):
        stars = n // 2 - 1
        R = -scale * torch.log((1.0 - _uniform(stars, g)) * (1.0 - _uniform(stars, g)))  # Sigma ~ exp(-R / scale)
        phi = 2.0 * math.pi * _uniform(stars, g)
        z = height * torch.atanh((2.0 * _uniform(stars, g) - 1.0).clamp(-0.999999, 0.999999))
        inside = centre + stars * (1.0 - (1.0 + R / scale) * torch.exp(-R / scale))
        vc = torch.sqrt(inside * R * R / (R * R + 40.0) ** 1.5)
        pos = torch.stack([R * torch.cos(phi), R * torch.sin(phi), z], 1)
        vel = torch.stack([-vc * torch.sin(phi), vc * torch.cos(phi), torch.zeros_like(z)], 1)
        if side > 0:
            t = math.radians(tilt)
            rot = torch.tensor([[1, 0, 0], [0, math.cos(t), -math.sin(t)], [0, math.sin(t), math.cos(t)]],
                               device="cuda", dtype=torch.float64)
            pos, vel = pos @ rot.T, vel @ rot.T
        zero = torch.zeros((1, 3), device="cuda", dtype=torch.float64)
        pos, vel = torch.cat([zero, pos]), torch.cat([zero, vel])
        pos[:, 0] += side * apart
        vel[:, 1] += side * speed
        mass = torch.ones(n // 2, device="cuda", dtype=torch.float64)
        mass[0] = centre
        halves.append((pos, vel, mass))
    return tuple(torch.cat(x) for x in zip(*halves))


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _bodies(case, seed):
    """float32 positions (n, 3), velocities (n, 3) and masses (n,) on the GPU."""
    g, n = _generator(seed), case["n"]
    if case["use"] == "ensemble":
        made = _plummer(_sizes(case), g, a=50.0)
    else:
        made = {"ball": lambda: _ball(n, g), "plummer": lambda: _plummer([n], g), "discs": lambda: _discs(n, g)}[
            case["shape"]]()
    return tuple(x.float() for x in made)


def _sizes(case):
    """An ensemble's system sizes, log-uniform (the seed makes the bodies, not the mix)."""
    rng = np.random.default_rng(2024 + case["n"])
    lo, hi = case["lo"], case["hi"]
    return [int(min(hi, x)) for x in np.floor(np.exp(rng.uniform(np.log(lo), np.log(hi + 1), case["n"])))]


def _vec4(x, pinned):
    """The reference's host layout: float32 (n, 4), w = 0; masses in column 0."""
    out = torch.zeros((x.shape[0], 4), dtype=torch.float32, pin_memory=pinned)
    if x.dim() == 1:
        out[:, 0] = x.cpu()
    else:
        out[:, :3] = x.cpu()
    return out.numpy()


def _system(pos, vel, mass, pinned):
    s = nb.ParticleSystem(_vec4(pos, pinned), _vec4(vel, pinned), _vec4(mass, pinned),
                          _vec4(torch.zeros_like(pos), pinned))
    s.forces = _vec4(torch.zeros_like(pos), pinned)
    return s


def _part(s, at, n):
    """Bodies at .. at + n of a system, in place."""
    return nb.ParticleSystem(s.positions[at:at + n], s.velocities[at:at + n], s.masses[at:at + n],
                             s.accelerations[at:at + n])


_stream = None


def _work_stream():
    """One stream for the program's work, as a caller with device buffers of its own would keep."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


# --------------------------------------------------------------- the cases
def prepare(case, seed):
    n = case["n"]
    pos, vel, mass = _bodies(case, seed)
    if case["use"] == "ensemble":
        return _prepare_ensemble(case, _system(pos, vel, mass, case["pinned"]))
    solver = nb.ParticleSolverCUDA(case["dt"], case["eps2"], n, mode=case["solver"], theta2=case["theta2"])
    solver.set_integrator(case["integrator"])
    solver.set_stream(_work_stream().cuda_stream)
    if case["solver"] == "bh":
        solver.set_key_mode(case["keys"])
    state = {"case": case, "solver": solver}
    if case["use"] == "forces":
        state["pos_mass"] = torch.cat([pos, mass[:, None]], 1).contiguous()
        state["force"] = torch.zeros((n, 4), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()  # made on torch's stream, read on the work stream
        return state
    state["system"] = _system(pos, vel, mass, case["pinned"])
    if case["use"] == "steps":
        zero = torch.zeros_like(pos)
        state["result"] = _system(zero, zero, zero[:, 0], case["pinned"])
    return state


def _prepare_ensemble(case, start):
    sizes = _sizes(case)
    ens = nb.Ensemble(crossover=CROSSOVER, pp_shape=PP_SHAPE, key_mode=case["keys"])
    ens.set_stream(_work_stream().cuda_stream)
    ids = [ens.add(n, case["dt"], case["eps2"], case["theta2"], integrator=case["integrator"]) for n in sizes]
    firsts = np.concatenate([[0], np.cumsum(sizes)])
    for sid, n, at in zip(ids, sizes, firsts):
        ens.upload(sid, _part(start, at, n))
    parts = [(sid, _part(start, at, n)) for sid, n, at in zip(ids, sizes, firsts)]
    return {"case": case, "ensemble": ens, "result": start, "parts": parts}


def run(state):
    case = state["case"]
    if case["use"] == "ensemble":
        ens, out = state["ensemble"], state["result"]
        ens.step(case["steps"], graph_steps=case["steps"])
        for sid, part in state["parts"]:
            ens.download(sid, part, masses=False)
        return {"positions": out.positions, "velocities": out.velocities, "accelerations": out.accelerations}
    solver = state["solver"]
    if case["use"] == "forces":
        call = solver.pp_forces_device if case["solver"] == "pp" else solver.bh_forces_device
        call(state["pos_mass"], state["force"])
        return {"forces": state["force"]}
    if case["use"] == "steps":
        s = state["result"]
        solver.upload(state["system"])
        solver.step(case["steps"])
        solver.download(s)
    else:
        s = state["system"]
        solver.update_particle_positions(s)
    return {"positions": s.positions, "velocities": s.velocities, "accelerations": s.accelerations,
            "forces": s.forces}


# --------------------------------------------------- what a pass has to do
def _evaluations(n, bh, theta2):
    """Pairwise evaluations of one force pass: every ordered pair, or what the opening criterion accepts (about 28
    log2(n) / theta^2 per body over the sizes here)."""
    return n * min(n, 28.0 * math.log2(max(n, 2)) / theta2) if bh else float(n) * n


def work(case):
    """20 operations per evaluation; positions, velocities, accelerations and masses read and the outputs written."""
    steps = case.get("steps", 1)
    if case["use"] == "ensemble":
        sizes = _sizes(case)
        flops = sum(20.0 * steps * _evaluations(n, n >= CROSSOVER, case["theta2"]) for n in sizes)
        return {"bytes": 96 * sum(sizes), "flops": flops}
    n, per_body = case["n"], 32 if case["use"] == "forces" else 128
    return {"bytes": per_body * n, "flops": 20.0 * steps * _evaluations(n, case["solver"] == "bh", case["theta2"])}


# -------------------------------------------------------- 64-bit reference
EXACT_PAIRS = 6e10  # beyond this a 64-bit direct sum takes too long


def _direct64(pos, mass, eps2):
    n = pos.shape[0]
    out = torch.empty_like(pos)
    rows = max(1, min(n, (1 << 25) // n))
    for i in range(0, n, rows):
        d = [pos[None, :, a] - pos[i:i + rows, None, a] for a in range(3)]
        r2 = d[0] * d[0]
        r2.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        w = torch.where(r2 > 0, r2 + eps2, torch.inf).rsqrt_()  # a body does not act on itself
        w = w * w * w * mass[None, :]
        for a in range(3):
            out[i:i + rows, a] = (d[a] * w).sum(1)
    return out


def _run64(pos, vel, mass, case, steps):
    dt = float(np.float32(case["dt"]))
    eps2 = float(np.float32(case["eps2"]))
    x, v, m = pos.double(), vel.double(), mass.double()
    a = torch.zeros_like(x)
    for _ in range(steps):
        f = _direct64(x, m, eps2)
        if case["integrator"] == "gpu_euler":
            v = v + f * dt
            x = x + v * dt
        else:
            v = v + a * (dt / 2)
            x = x + v * dt
            v = v + f * (dt / 2)
        a = f
    return x, v, a


def _pad(x):
    return torch.cat([x, torch.zeros_like(x[:, :1])], 1).cpu().numpy()


def exact(case, seed):
    """The direct sum in 64 bits (Barnes-Hut approximates it to its opening angle), and the steps it drives."""
    steps = case.get("steps", 1)
    sizes = _sizes(case) if case["use"] == "ensemble" else [case["n"]]
    if steps * sum(float(n) * n for n in sizes) > EXACT_PAIRS:
        return None
    pos, vel, mass = _bodies(case, seed)
    if case["use"] == "forces":
        return {"forces": _pad(_direct64(pos.double(), mass.double(), float(np.float32(case["eps2"]))))}
    parts = [_run64(p, v, m, case, steps) for p, v, m in zip(pos.split(sizes), vel.split(sizes), mass.split(sizes))]
    x, v, a = (_pad(torch.cat(p)) for p in zip(*parts))
    out = {"positions": x, "velocities": v, "accelerations": a}
    return out if case["use"] == "ensemble" else {**out, "forces": a}
