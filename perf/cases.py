"""Performance cases of the simulation engine: what a user's program has it do.

Every case is one call sequence through the public Python entry points
(:class:`pyrdsim_gb300.engine.Engine`, :func:`pyrdsim_gb300.adjoint.trajectory_loss`)
on inputs made from a seed: runs of the benchmark configurations at their own
sizes and at smaller, larger and odd ones (both force precisions, with and
without reactions, bonds, walls, trajectory frames, batching, 2D and 3D), the
gradient of a trajectory loss, and the analysis of stored configurations
(observables, g(r) histograms, neighbour pairs).  ``listed`` names the cases
that are reported, ``draw`` gives others of the same ranges, ``work`` counts
the bytes and operations a case cannot do without and ``exact`` restates the
small ones in float64 with plain numpy and torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pyrdsim_gb300 import model, workloads
from pyrdsim_gb300.adjoint import Adjoint, trajectory_loss
from pyrdsim_gb300.engine import Engine

LJ_R0 = workloads.WCA_R0


def listed():
    return [
        # an interactive user's small box: the LJ fluid configuration, where
        # one step is all latency
        run_case("lj_fluid_1k", "lj2d", n=1024, steps=100),
        # the same configuration by the plain float64 method
        run_case("lj_fluid_1k_float64", "lj2d", n=1024, steps=50, precision="float64"),
        # a production run that stores a frame every 10 steps (an odd size,
        # three species, an inhibited reaction)
        run_case("inhibited_5k_frames", "inhibited", n=5003, steps=100, stride=10),
        # a 3D fluid: long neighbour lists
        run_case("lj_fluid_3d_14k", "lj3d", n=13824, steps=50),
        # the benchmark's configuration, end to end: host state in, a segment
        # of the run, host state out, at the benchmark's list period
        run_case("wall_fluid_65k", "wall", n=65536, steps=200, list_period=20, reload=True),
        # bonded molecules: the three-patch colloids
        run_case("patchy_65k", "patchy", n=65536, steps=100),
        # replicas of uneven size (LJ and long-ranged Yukawa) in one batch
        run_case("ensemble_64", "ensemble", n=64, steps=50),
        # the largest box: far more particles than fit the chip at once
        run_case("wall_fluid_1m", "wall", n=1048576, steps=40),
        # fitting force-field parameters: loss and gradients of short windows
        adjoint_case("adjoint_1k", n=1001, steps=16, loss_steps=8, checkpoint_every=8),
        adjoint_case("adjoint_16k", n=16384, steps=32, loss_steps=16, checkpoint_every=32),
        # analysis of a stored frame: energies, virial and g(r)
        {"name": "observe_65k", "kind": "observe", "n": 65536, "r_max": 5.0, "bins": 200},
        # the neighbour pairs of a stored frame
        {"name": "pairs_16k", "kind": "pairs", "n": 16384},
    ]


def run_case(name, system, n, steps, precision="float32", list_period=0, stride=0, reload=False):
    """``steps`` steps of a system of ``n`` particles (ensemble: systems);
    stride > 0 keeps a trajectory frame every ``stride`` steps; reload sets
    the state from host memory first."""
    c = {"kind": "run", "system": system, "n": n, "steps": steps, "precision": precision,
         "list_period": list_period, "stride": stride, "reload": reload}
    return dict(c, name=name) if name else c


def adjoint_case(name, n, steps, loss_steps, checkpoint_every):
    c = {"kind": "adjoint", "n": n, "steps": steps, "loss_steps": loss_steps,
         "checkpoint_every": checkpoint_every}
    return dict(c, name=name) if name else c


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lj2d", "lj2d", "float64", "lj3d", "wall", "wall", "patchy", "ensemble",
                       "inhibited", "adjoint", "observe", "pairs"])
    if kind == "adjoint":
        e = rng.choice([8, 16, 32])
        t = rng.randint(8, 32)
        return adjoint_case("", log_uniform(rng, 300, 16384), t, rng.randint(1, t), e)
    if kind == "observe":
        return {"kind": "observe", "n": log_uniform(rng, 1000, 131072),
                "r_max": round(rng.uniform(2.0, 6.0), 3), "bins": rng.randint(50, 400)}
    if kind == "pairs":
        return {"kind": "pairs", "n": log_uniform(rng, 500, 32768)}
    if kind == "ensemble":
        return run_case("", "ensemble", rng.randint(3, 64), rng.randint(20, 50))
    if kind == "float64":
        return run_case("", "lj2d", log_uniform(rng, 256, 16384), rng.randint(20, 100),
                        precision="float64")
    n = {"lj2d": log_uniform(rng, 256, 262144), "lj3d": round(log_uniform(rng, 8, 36)) ** 3,
         "wall": log_uniform(rng, 2048, 1048576), "patchy": 4 * log_uniform(rng, 256, 40000),
         "inhibited": log_uniform(rng, 512, 65536)}[kind]
    # the same particle-steps as the largest listed case at most
    steps = min(rng.randint(30, 300), 40 * 1048576 // n)
    stride = rng.choice([0, 0, 10, 25]) if n <= 65536 else 0
    return run_case("", kind, n, steps if kind != "lj3d" else min(steps, 50),
                    # the inhibited deck's rs leaves no room for a longer period's skin
                    list_period=0 if kind == "inhibited" else rng.choice([0, 0, 20]),
                    stride=stride, reload=rng.random() < 0.3)


# ---- inputs -------------------------------------------------------------

def lj_fluid_3d(n, rho, seed, dt=1e-4):
    """The LJ fluid configuration in a periodic cube, jittered-lattice start."""
    rng = np.random.default_rng(seed)
    side = int(round(n ** (1.0 / 3.0)))
    L = float((n / rho) ** (1.0 / 3.0))
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    x = (g + 0.5 + rng.uniform(-0.08, 0.08, g.shape)) * (L / side)
    m = model.Model.from_dict({
        "n_dim": 3, "l": np.array([L] * 3), "periodic": np.ones(3), "dt": dt, "n_steps": 10000,
        "n_out": 100000, "tau_by_taud": np.array([1.0]), "seed": seed,
        "interactions": [{"type": "lj", "pair": [0, 0], "u0": 1.0, "r0": LJ_R0, "rc": 2.5,
                          "n": 6}], "reactions": []})
    return single_atoms(m, x, np.zeros(len(x), np.int32))


def single_atoms(m, x, types):
    n = len(x)
    mol = np.stack([np.arange(n), np.zeros(n, int), np.zeros(n, int)], 1).astype(np.int32)
    return model.SystemData(m, x, types, mol, np.arange(n, dtype=np.int32))


def ensemble(n_systems, seed, dt=1e-4):
    """Independent systems of 256 to 16,384 particles (sizes spread evenly
    over their logarithm), LJ and Yukawa in turn, every other pair of them
    with a two-state reaction; densities and temperatures from the seed."""
    rng = np.random.default_rng(seed)
    out = []
    for s in range(n_systems):
        n = int(256 * 64 ** (s / max(1, n_systems - 1)))
        rho, kT = rng.uniform(0.2, 0.7), rng.uniform(0.5, 2.0)
        L = float(np.sqrt(n / rho))
        law = ({"type": "lj", "r0": LJ_R0, "rc": 2.5, "n": 6, "u0": 1.0 / kT} if s % 2 == 0 else
               {"type": "yukawa", "r0": 1.0, "rc": 5.0, "u0": 10.0 / kT})
        nt = 2 if s % 4 < 2 else 1
        reactions = [] if nt == 1 else [
            {"type": "linear", "reactant": a, "product": 1 - a, "rate": rng.uniform(0.01, 1)}
            for a in (0, 1)]
        m = model.Model.from_dict({
            "n_dim": 2, "l": np.array([L, L]), "periodic": np.ones(2), "dt": dt, "n_steps": 5000,
            "n_out": 1000000, "tau_by_taud": np.full(nt, kT), "seed": int(rng.integers(1, 2**31)),
            "interactions": [dict(law, pair=[a, b]) for a in range(nt) for b in range(a, nt)],
            "reactions": reactions})
        x = workloads.jittered_lattice(n, [L, L], rng)
        out.append(single_atoms(m, x, rng.integers(0, nt, n).astype(np.int32)))
    return out


def systems_of(case, seed):
    n, system = case["n"], case.get("system", "wall")
    if system == "lj2d":
        return [workloads.lj_fluid(n=n, seed=seed, start="lattice")]
    if system == "lj3d":
        return [lj_fluid_3d(n, 0.5, seed)]
    if system == "patchy":
        return [workloads.patchy_colloids(n_molecules=n // 4, seed=seed)]
    if system == "inhibited":
        return [workloads.inhibited_mixture(n=n, seed=seed)]
    if system == "ensemble":
        return ensemble(n, seed)
    return [workloads.active_wall_fluid(n=n, seed=seed)]


def pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def mean_pairs(n):
    """Pairs of the wall fluid (density 0.4) within its neighbour radius 5."""
    return 0.5 * n * 0.4 * math.pi * 5.0 ** 2


def prepare(case, seed):
    if case["kind"] == "adjoint":
        w = workloads.mixed_lj_yukawa(n=case["n"], seed=seed)
        adj = Adjoint(2, w["L"], w["dt"], w["mobility"], w["types"],
                      workloads.mixed_lj_yukawa_laws(w), loss_steps=case["loss_steps"],
                      checkpoint_every=case["checkpoint_every"])
        x0 = torch.tensor(w["x0"], device="cuda", requires_grad=True)
        params = torch.tensor(workloads.mixed_lj_yukawa_params(w["theta"]), requires_grad=True)
        return {"case": case, "adj": adj, "x0": x0, "params": params,
                "xi": adjoint_noise(case, seed).cuda()}
    sds = systems_of(case, seed)
    eng = Engine(sds, precision=case.get("precision", "float32"),
                 list_period=case.get("list_period", 0))
    s = {"case": case, "engine": eng}
    if case["kind"] != "run" or case["reload"]:  # host state, as read from a file
        x = np.concatenate([d.x for d in sds])
        t = np.concatenate([d.types for d in sds])
        s["x_in"], s["t_in"] = pinned(x.shape, torch.float64), pinned(t.shape, torch.int32)
        s["x_in"][:], s["t_in"][:] = x, t
    if case["kind"] == "pairs":  # room for the pairs of any start: 25 % above the mean
        s["pairs"] = np.empty((int(1.25 * mean_pairs(case["n"])) + 64, 2), np.int32)
    if case["kind"] == "run":
        s["x"], s["t"] = pinned((eng.N, eng.D), torch.float64), pinned((eng.N,), torch.int32)
        if case["stride"]:
            eng.set_trajectory(case["stride"], max(1, case["steps"] // case["stride"]))
    return s


def run(s):
    case = s["case"]
    if case["kind"] == "adjoint":
        loss = trajectory_loss(s["x0"], s["params"], s["xi"], s["adj"])
        gx, gp = torch.autograd.grad(loss, (s["x0"], s["params"]))
        return {"loss": loss.detach(), "grad_x0": gx, "grad_params": gp}
    eng = s["engine"]
    if "x_in" in s:
        eng.set_state(s["x_in"], s["t_in"])
    if case["kind"] == "observe":
        out = eng.observables()
        out["type_counts"] = np.array(out["type_counts"])
        out["rdf_counts"] = eng.rdf_counts(case["r_max"], n_bins=case["bins"])
        return out
    if case["kind"] == "pairs":
        p = eng.pairs()
        s["pairs"][:len(p)], s["pairs"][len(p):] = p, -1
        return {"pairs": s["pairs"], "count": len(p)}
    eng.step(case["steps"])
    x, t = eng.state(s["x"], s["t"])
    out = {"x": x, "types": t}
    if case["stride"]:
        out["frames"], out["frame_types"] = eng.trajectory()
    return out


# ---- what a pass cannot do without ---------------------------------------

def work(case):
    """Bytes: inputs and outputs once, for steps the state read and written
    once per step (16 B of position per dimension pair and 4 B of type each
    way).  Flops: about 30 per pair inside the cutoff and 120 per particle and
    step (noise, update); gradients three times the steps."""
    n = case["n"]
    if case["kind"] == "adjoint":
        # 9 neighbours within the LJ cutoff, half of them Yukawa partners too
        flops = n * case["steps"] * (2 + 3) * 11 * 30.0
        return {"bytes": n * 16.0 * (case["steps"] + 3), "flops": flops}
    if case["kind"] == "observe":
        pairs = 0.5 * n * 0.4 * math.pi * case["r_max"] ** 2
        return {"bytes": n * 20.0 + 8.0 * case["bins"], "flops": pairs * 10.0}
    if case["kind"] == "pairs":
        return {"bytes": n * 20.0 + 8.0 * mean_pairs(n), "flops": mean_pairs(n) * 10.0}
    system, d = case["system"], 3 if case["system"] == "lj3d" else 2
    if system == "ensemble":
        n = sum(int(256 * 64 ** (s / max(1, case["n"] - 1))) for s in range(case["n"]))
    near = {"lj2d": 9.8, "lj3d": 32.0, "wall": 4.0, "patchy": 6.0, "ensemble": 22.0,
            "inhibited": 4.0}[system]
    return {"bytes": n * case["steps"] * (16.0 * d + 8.0),
            "flops": n * case["steps"] * (30.0 * near + 120.0)}


# ---- float64 restatements -------------------------------------------------

def exact(case, seed):
    if case["kind"] == "adjoint":
        return exact_adjoint(case, seed) if case["n"] <= 1100 else None
    if case["kind"] == "observe":
        return exact_observe(case, seed)
    if case["kind"] != "run" or case["system"] not in ("lj2d", "lj3d"):
        return None
    if float(case["n"]) ** 2 * case["steps"] > 1e10:
        return None
    return exact_lj(case, seed)


def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def philox(step, n, tag, seed):
    """Philox4x32-10 (Salmon et al., SC'11) words of particles 0 .. n-1."""
    mask = np.uint64(0xFFFFFFFF)
    c = [np.full(n, step & 0xFFFFFFFF, np.uint64), np.full(n, step >> 32, np.uint64),
         np.arange(n, dtype=np.uint64), np.full(n, tag, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask,
             (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def normals(step, n, d, seed):
    """The normals of one step: Box-Muller on the words' float32 uniforms."""
    w = philox(step, n, 0, seed)
    f32 = [v.astype(np.float32) * np.float32(2.0 ** -32) for v in w]
    out = []
    for a, b in ((0, 1), (2, 3)):
        r = np.sqrt(-2.0 * np.log((f32[a] + np.float32(2.0 ** -33)).astype(np.float64)))
        phi = 2.0 * np.pi * f32[b].astype(np.float64)
        out += [r * np.cos(phi), r * np.sin(phi)]
    return np.stack(out[:d], 1)


def row_chunks(n, most=1 << 25):
    rows = max(1, min(n, most // n))
    return [(a, min(a + rows, n)) for a in range(0, n, rows)]


def exact_lj(case, seed):
    sd = systems_of(case, seed)[0]
    m, dev = sd.model, device()
    x = torch.tensor(sd.x, device=dev)
    n, d = x.shape
    L = torch.tensor(np.asarray(m.L), device=dev)
    frames = []
    for step in range(1, case["steps"] + 1):
        a = torch.zeros_like(x)
        for b, e in row_chunks(n):
            dx = x[None, :, :] - x[b:e, None, :]
            dx -= L * torch.round(dx / L)
            r2 = (dx * dx).sum(-1)
            r2[torch.arange(e - b), torch.arange(b, e)] = 1e9
            s = (LJ_R0 * LJ_R0 / r2) ** 3
            f = torch.where(r2 <= 2.5 ** 2, -12.0 * s * (s - 1.0) / r2, torch.zeros_like(r2))
            a[b:e] = (f[:, :, None] * dx).sum(1)
        xi = torch.tensor(normals(step, n, d, m.seed), device=dev)
        x = torch.remainder(x + m.dt * a + math.sqrt(2.0 * m.dt) * xi, L)
        if case["stride"] and step % case["stride"] == 0:
            frames.append(x.cpu().numpy())
    out = {"x": x.cpu().numpy(), "types": None}
    if case["stride"]:
        out["frames"] = np.stack(frames) if frames else np.zeros((1, n, d))
        out["frame_types"] = None
    return out


def lj_potential(r2, r0=LJ_R0):
    s = (r0 * r0 / r2) ** 3
    return s * (s - 2.0), 12.0 * s * (s - 1.0)  # U, -r dU/dr


def exact_observe(case, seed):
    sd = systems_of(case, seed)[0]
    dev = device()
    if sd.x.shape[0] > 20000 and dev.type != "cuda":
        return None
    x, t = torch.tensor(sd.x, device=dev), torch.tensor(sd.types, device=dev)
    n, L = x.shape[0], float(sd.model.L[0])
    wca2, rc2, ymin2 = LJ_R0 ** 2, 2.5 ** 2, math.inf
    energy = torch.zeros((), dtype=torch.float64, device=dev)
    virial = torch.zeros((), dtype=torch.float64, device=dev)
    for b, e in row_chunks(n):
        dx = x[None, :, 0] - x[b:e, None, 0]
        dx -= L * torch.round(dx / L)
        dy = x[None, :, 1] - x[b:e, None, 1]
        r2 = dx * dx + dy * dy
        r2[torch.arange(e - b), torch.arange(b, e)] = 1e9
        ymin2 = min(ymin2, float(r2.min()))
        active = (t[b:e, None] == 1) & (t[None, :] == 1)
        near = r2 <= torch.where(active, rc2, wca2)
        U, W = lj_potential(r2[near])
        energy += 0.5 * U.sum()
        virial += 0.5 * W.sum()
    y = x[:, 1]
    cut = torch.where(t == 1, 2.5, 0.4 ** (1.0 / 6.0))
    s3 = (1.0 / y) ** 3
    wall = torch.where(y <= cut, 2.0 / 15.0 * s3 ** 3 - s3, torch.zeros_like(y)).sum()
    out = dict.fromkeys(("bond_energy", "angle_energy", "n_pairs", "n_particles", "type_counts",
                         "rdf_counts"))
    out.update(pair_energy=float(energy), virial=float(virial), wall_energy=float(wall),
               min_distance=math.sqrt(ymin2))
    return out


def adjoint_noise(case, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn((case["steps"], case["n"], 2), dtype=torch.float64, generator=g)


def exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint
    dev = device()
    w = workloads.mixed_lj_yukawa(n=case["n"], seed=seed)
    x0 = torch.tensor(w["x0"], device=dev, requires_grad=True)
    params = torch.tensor(workloads.mixed_lj_yukawa_params(w["theta"]), device=dev,
                          requires_grad=True)
    t = torch.tensor(w["types"], device=dev)
    L, dt, N = float(w["L"][0]), w["dt"], case["n"]
    lo, hi = torch.minimum(t[:, None], t[None, :]), torch.maximum(t[:, None], t[None, :])
    eye = torch.eye(N, dtype=torch.bool, device=dev)
    laws = [("lj", a, b, w["rc_lj"]) for a, b in w["pairs"]] + [("yukawa", 1, 1, w["rc_yukawa"])]

    def law(kind, u0, r0, r):  # U, dU/dr
        if kind == "lj":
            s = (r0 / r) ** 6
            return u0 * s * (s - 2.0), -12.0 * u0 * s * (s - 1.0) / r
        e = torch.exp(-r / r0)
        return u0 * e / r, -u0 * e * (1.0 / (r * r0) + 1.0 / (r * r))

    def state(x, p):  # drift and U + W / (d V)
        d = x[None, :, :] - x[:, None, :]
        d = d - L * torch.round(d / L)
        r = torch.sqrt((d * d).sum(-1) + eye.double())
        f, q = torch.zeros_like(r), torch.zeros((), dtype=torch.float64, device=dev)
        for k, (kind, a, b, rc) in enumerate(laws):
            m = (lo == a) & (hi == b) & ~eye & (r < rc)
            U, fr = law(kind, p[k, 0], p[k, 1], r)
            Uc = law(kind, p[k, 0], p[k, 1], torch.tensor(rc, dtype=torch.float64, device=dev))[0]
            f = f + torch.where(m, fr / r, torch.zeros_like(r))
            q = q + 0.5 * torch.where(m, U - Uc - r * fr / (2 * L * L), torch.zeros_like(r)).sum()
        return (f[:, :, None] * d).sum(1), q

    xi = adjoint_noise(case, seed).to(dev)
    T, K = case["steps"], case["loss_steps"]
    x, loss = x0, 0.0
    for n in range(T + 1):
        a, q = checkpoint(state, x, params, use_reentrant=False)
        if n >= T - K + 1:
            loss = loss + q / K
        if n < T:
            x = torch.remainder(x + dt * a + math.sqrt(2.0 * dt) * xi[n], L)
    gx, gp = torch.autograd.grad(loss, (x0, params))
    return {"loss": loss.detach(), "grad_x0": gx, "grad_params": gp}
