"""The work a user of mdtk_b200 has it do, as a list of cases to be timed and
compared: force calls, device-resident runs, host-driven steps, batches of
impacts and adjoint gradients, through the package's public entry points.

listed() names one case per use; draw() gives further ones of the same ranges;
prepare() builds what a program holds before the call (a context with a loaded
system), run() is one pass, work() the least a pass has to move and compute,
and exact() the outputs in plain numpy and torch where that is short to write.
"""
import math

import numpy as np
import torch

import mdtk_b200 as M
from mdtk_b200 import builders as B

POTENTIALS = {
    "rebo": M.POT_REBO,
    "rebo_tors": M.POT_REBO | M.POT_ETORS,
    "airebo": M.POT_AIREBO,
    "brenner": M.POT_BRENNER,
    "airebo_metal": M.POT_AIREBO | M.POT_METAL,
}
PRECISIONS = {"fp64": M.PREC_FP64, "mixed": M.PREC_FP32_MIXED}


def listed():
    return [
        # FProxy's force call on the reference's own example molecule
        # (examples/C2H6): the smallest call, all latency.
        dict(name="c2h6_force", use="force", system="c2h6", size=1, potential="rebo_tors", precision="fp64"),
        # A small liquid in an unchanged host program: the state crosses to
        # the device and back every step (mdg_step_host, one step a call).
        dict(name="ethane_240_host_step", use="host", system="ethane", size=30, potential="airebo",
             precision="fp64", steps=1, dt=0.25),
        # Plain REBO carbon NVE: the 1,728-atom diamond at 300 K with its
        # per-step energies, in stretches of 40 steps.
        dict(name="diamond_1728_rebo_run", use="run", system="diamond", size=6, potential="rebo",
             precision="fp64", steps=40, dt=0.5, energies=True),
        # The same crystal with first-generation Brenner, set 2, at an odd size.
        dict(name="diamond_1000_brenner_run", use="run", system="diamond", size=5, potential="brenner",
             precision="fp64", steps=40, dt=0.5, energies=True, brenner_set=2),
        # The force call of the drop-in classes under a host-side SimLoop:
        # new positions in, energies and gradient out, 8,832 atoms.
        dict(name="ethane_8832_force", use="force", system="ethane", size=92, tiles=12, potential="airebo",
             precision="fp64"),
        # The hydrocarbon liquid of the headline configuration (5,460
        # molecules), device-resident, 40 steps between looks at the state.
        dict(name="ethane_43680_run", use="run", system="ethane", size=91, tiles=60, potential="airebo",
             precision="fp64", steps=40, dt=0.25, energies=False),
        # The FP32-mixed mode on the liquid, with per-step energies; the work
        # split is fixed so that runs of one program can be repeated exactly.
        dict(name="ethane_16128_mixed_run", use="run", system="ethane", size=84, tiles=24, potential="airebo",
             precision="mixed", steps=40, dt=0.25, energies=True, task_mode=2),
        # The large crystal of the precision study: 40^3 cells, 600 K.
        dict(name="diamond_512000_mixed_run", use="run", system="hot_diamond", size=40, potential="airebo",
             precision="mixed", steps=6, dt=0.5, energies=False, task_mode=2),
        # 64 cluster impacts on graphite slabs of 800 to 6,000 atoms in one
        # context, energies of each system at each step.
        dict(name="impacts_64_mixed_batch", use="batch", system="impact", size=64, potential="airebo",
             precision="mixed", steps=6, dt=0.2, task_mode=2),
        # mdtrajsim's way of running: many small impacts together, adaptive
        # time step, a thermal bath at the slab's edge.
        dict(name="small_impacts_64_bath_run", use="run", system="small_impacts", size=64, potential="airebo",
             precision="fp64", steps=40, dt=0.2, energies=False, bath=True),
        # A metal slab under an ion, ethane molecules above it: the whole
        # potential set of the applications.
        dict(name="cu_slab_19233_run", use="run", system="cu_slab", size=24, potential="airebo_metal",
             precision="fp64", steps=20, dt=0.25, energies=True),
        # Gradient of a trajectory loss (parameters, initial state): forward
        # and backward over 10 steps with checkpoints.
        dict(name="diamond_1000_adjoint", use="adjoint", system="hot_diamond", size=5, potential="airebo",
             precision="fp64", steps=10, dt=0.5, task_mode=1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _liquid(rng, tiles):
    """Size and tiles of a drawn liquid: a cell of 28 to 108 molecules, repeated."""
    size = rng.choice([rng.randint(28, 32), rng.randint(58, 64), rng.randint(81, 108)])
    return dict(system="ethane", size=size, tiles=_log_int(rng, 1, tiles))


def draw(rng):
    use = rng.choice(["force", "host", "run", "mixed", "crystal", "brenner", "batch", "bath", "metal", "adjoint"])
    if use == "force":
        return dict(use="force", precision="fp64", potential=rng.choice(["rebo", "rebo_tors", "airebo"]),
                    **_liquid(rng, 30))
    if use == "host":
        return dict(use="host", potential="airebo", precision="fp64", steps=rng.randint(1, 10), dt=0.25,
                    **_liquid(rng, 30))
    if use == "run":
        return dict(use="run", potential="airebo", precision="fp64", steps=rng.randint(10, 40), dt=0.25,
                    energies=rng.random() < 0.5, **_liquid(rng, 55))
    if use == "mixed":
        return dict(use="run", system="hot_diamond", size=_log_int(rng, 4, 32), potential="airebo",
                    precision="mixed", steps=rng.randint(4, 8), dt=0.5, energies=rng.random() < 0.5,
                    task_mode=rng.randint(1, 3))
    if use == "crystal":
        return dict(use="run", system="diamond", size=_log_int(rng, 3, 24), potential="rebo", precision="fp64",
                    steps=rng.randint(10, 40), dt=0.5, energies=rng.random() < 0.5)
    if use == "brenner":
        return dict(use="run", system="diamond", size=_log_int(rng, 3, 20), potential="brenner", precision="fp64",
                    steps=rng.randint(10, 40), dt=0.5, energies=rng.random() < 0.5, brenner_set=rng.randint(1, 2))
    if use == "batch":
        return dict(use="batch", system="impact", size=rng.randint(2, 48), potential="airebo", precision="mixed",
                    steps=rng.randint(2, 8), dt=0.2, task_mode=rng.randint(1, 3))
    if use == "bath":
        return dict(use="run", system="small_impacts", size=rng.randint(2, 96), potential="airebo",
                    precision="fp64", steps=rng.randint(10, 40), dt=0.2, energies=False, bath=True)
    if use == "metal":
        return dict(use="run", system="cu_slab", size=rng.randint(8, 24), potential="airebo_metal",
                    precision="fp64", steps=rng.randint(10, 20), dt=0.25, energies=rng.random() < 0.5)
    return dict(use="adjoint", system="hot_diamond", size=rng.randint(4, 8), potential="airebo", precision="fp64",
                steps=rng.randint(4, 12), dt=0.5, task_mode=rng.randint(1, 3))


# ---------------------------------------------------------------- systems


def _tiled_liquid(size, tiles, seed, rng):
    """An ethane liquid at 0.55 g/cm^3 and 300 K from a cell of `size`
    molecules repeated `tiles` times, every atom displaced on its own."""
    s = B.ethane_liquid(size, density_g_cm3=0.55, temp_k=300.0, seed=seed)
    if tiles == 1:
        return s
    reps = [1, 1, tiles]
    for a in range(1, int(round(tiles ** (1 / 3))) + 1):  # the most cubic block of cells
        for b in range(a, int(math.sqrt(tiles / a)) + 1):
            if tiles % (a * b) == 0:
                reps = [a, b, tiles // (a * b)]
    shifts = np.stack(np.meshgrid(*map(np.arange, reps), indexing="ij"), -1).reshape(-1, 1, 3) * s["box"]
    pos = (s["pos"][None] + shifts).reshape(-1, 3)
    s["pos"] = pos + rng.normal(scale=0.02, size=pos.shape)
    s["z"] = np.tile(s["z"], tiles)
    s["fixed"] = np.tile(s["fixed"], tiles)
    s["vel"] = B.thermal_velocities(s["z"], 300.0, rng)
    s["box"] = s["box"] * reps
    s["pos"] = np.mod(s["pos"], s["box"])
    return s


def _system(case, seed):
    """The atoms of a case (a dict as the builders return), or a list of them."""
    kind, size = case["system"], case["size"]
    rng = np.random.default_rng(seed)
    if kind == "c2h6":
        s = B.c2h6_example()
        s["pos"] = s["pos"] + rng.normal(scale=0.02, size=s["pos"].shape)
        return s
    if kind == "ethane":
        return _tiled_liquid(size, case.get("tiles", 1), seed, rng)
    if kind == "diamond":
        return B.diamond(size, temp_k=300.0, seed=seed)
    if kind == "hot_diamond":
        return B.diamond(size, temp_k=600.0, disp_sigma=0.05, seed=seed)
    if kind == "impact":
        # sizes and impact energies go by the system's place, the state by the seed
        out = B.impact_batch(size)
        for s in out:
            s["pos"] = s["pos"] + rng.normal(scale=0.02, size=s["pos"].shape)
            s["vel"][:-13] = B.thermal_velocities(s["z"][:-13], 300.0, rng, s["fixed"][:-13])
        return out
    if kind == "small_impacts":
        out = []
        for k in range(size):
            slab = B.graphite_slab(2, 8, 4, temp_k=300.0, seed=seed + k)
            x, y = rng.uniform(0, slab["box"][0]), rng.uniform(0, slab["box"][1])
            out.append(B.add_atoms(slab, [6], [[x, y, slab["pos"][:, 2].max() + 3.0]], vel=[[0, 0, -0.04]]))
        return out
    if kind == "cu_slab":
        cu = B.fcc(29, size, size, max(4, size // 3), pbc=(1, 1, 0), temp_k=300.0, seed=seed)
        top, edge = cu["pos"][:, 2].max(), cu["box"][0]
        mol = B.c2h6_example()
        m = int((edge - 1.0) // 8.5)
        zs, ps = [], []
        for i in range(m):
            for j in range(m):
                zs.append(mol["z"])
                ps.append(mol["pos"] - mol["pos"].mean(axis=0) + [4.0 + 8.5 * i, 4.0 + 8.5 * j, top + 3.0])
        zs.append(np.array([18], np.int32))
        ps.append(np.array([[edge / 2, edge / 2, top + 8.0]]))
        s = B.add_atoms(cu, np.concatenate(zs), np.concatenate(ps))
        s["vel"][-1] = [0.0, 0.0, -0.05]
        return s
    raise ValueError(kind)


def _load(case, system):
    caps = {k: case[k] for k in ("task_mode",) if k in case}
    ctx = M.Context(potentials=POTENTIALS[case["potential"]], precision=PRECISIONS[case["precision"]],
                    brenner_set=case.get("brenner_set", 1), **caps)
    if isinstance(system, list):
        ctx.set_batch(system)
    else:
        ctx.set_system(system["z"], system["pos"], system["vel"], system["box"], system["pbc"], system["fixed"])
    return ctx


def prepare(case, seed):
    system = _system(case, seed)
    st = {"case": case, "ctx": _load(case, system)}
    rng = np.random.default_rng(seed + 1)
    if case["use"] == "force":
        # two frames of the same trajectory, taken in turn as a host loop would
        pos = system["pos"]
        st["frames"] = [pos, pos + rng.normal(scale=0.005, size=pos.shape)]
        st["next"] = 0
    elif case["use"] == "host":
        st["pos"], st["vel"] = system["pos"].copy(), system["vel"].copy()
    elif case["use"] == "adjoint":
        n = len(system["z"])
        st["seed_pos"] = rng.normal(scale=0.02 / n, size=(n, 3))
        st["seed_vel"] = rng.normal(scale=0.02 / n, size=(n, 3))
        st["start"] = system["pos"], system["vel"]
    if case.get("bath"):
        st["ctx"].set_thermal_bath(M.TB_BOX, 300.0, 1e13 * 1e-15, [-10.0, 3.0, 1.0])
        st["ctx"].set_adaptive_dt(True, 1.0, case["dt"])
    return st


# ---------------------------------------------------------------- one pass


def run(state):
    case, ctx = state["case"], state["ctx"]
    use = case["use"]
    if use == "force":
        ctx.set_state(state["frames"][state["next"]])
        state["next"] ^= 1
        e, terms, grad = ctx.compute()
        return {"energy": e, "terms": terms, "grad": grad}
    if use == "host":
        epot, etot = ctx.step_host(case["steps"], case["dt"], state["pos"], state["vel"])
        return {"epot": epot, "etot": etot, "pos": state["pos"], "vel": state["vel"]}
    if use == "batch":
        epot, etot = ctx.batch_run(case["steps"], case["dt"])
        pos, vel, image = ctx.get_state()
        return {"epot": epot, "etot": etot, "pos": pos, "vel": vel, "image": image}
    if use == "adjoint":
        ctx.set_state(*state["start"])
        pos, vel, epot = ctx.adjoint_forward(case["steps"], case["dt"], 5)
        grad_params, grad_pos, grad_vel = ctx.adjoint_backward(state["seed_pos"], state["seed_vel"], 1e-5)
        return {"pos": pos, "vel": vel, "epot": epot, "grad_params": grad_params, "grad_pos": grad_pos,
                "grad_vel": grad_vel}
    energies = ctx.run(case["steps"], case["dt"], energies=case["energies"])
    pos, vel, image = ctx.get_state()
    out = {"pos": pos, "vel": vel, "image": image}
    if case["energies"]:
        out["epot"], out["etot"] = energies
    if case.get("bath"):
        out["time"], out["dt"] = ctx.get_time()
    return out


# ---------------------------------------------------------------- the least a pass costs


def _atoms(case):
    size = case["size"]
    kind = case["system"]
    if kind == "c2h6":
        return 8
    if kind == "ethane":
        return 8 * size * case.get("tiles", 1)
    if kind in ("diamond", "hot_diamond"):
        return 8 * size ** 3
    if kind == "impact":
        return 3580 * size  # the builder's mean
    if kind == "small_impacts":
        return 257 * size
    m = int((3.615 * size - 1.0) // 8.5)
    return 4 * size * size * max(4, size // 3) + 8 * m * m + 1


# Operations an atom's share of one energy and gradient needs (add and
# multiply 1, divide and root 4, exponential and cosine 12): bond-order terms
# by bonds and angles per atom, LJ terms by pairs within the cutoff.
_FLOPS = {
    ("ethane", "rebo"): 2.6e3, ("ethane", "rebo_tors"): 3.0e3, ("ethane", "airebo"): 1.3e4,
    ("c2h6", "rebo_tors"): 3.0e3,
    ("diamond", "rebo"): 5.0e3, ("diamond", "brenner"): 4.0e3,
    ("hot_diamond", "airebo"): 3.0e4, ("impact", "airebo"): 2.0e4, ("small_impacts", "airebo"): 1.5e4,
    ("cu_slab", "airebo_metal"): 5.0e3,
}


def work(case):
    n = _atoms(case)
    flops = _FLOPS[case["system"], case["potential"]] * n
    if case["use"] == "force":
        return {"bytes": 48.0 * n, "flops": flops}  # positions in, gradient out
    state = 48.0 * n  # positions and velocities
    if case["use"] == "adjoint":
        # start and loss seeds in, final state and its gradient out; forward,
        # recomputed segment, and one derivative pass of about three evaluations a step
        return {"bytes": 4 * state, "flops": 5 * flops * case["steps"]}
    return {"bytes": 2 * state, "flops": flops * case["steps"]}


# ---------------------------------------------------------------- 64-bit values

_EV_AMU = 1.6021e-12 / 1.6605655e-24 * 1e16 / 1e30  # 1 eV/amu in (Angstrom/fs)^2
_MASS_C = 12.0

# G_C2(cos theta) of REBO: value, slope and curvature at the knots
_G_KNOTS = [(-1.0, -0.010000, 0.104000, 0.000000), (-2.0 / 3.0, 0.028207, 0.131443, 0.140229),
            (-1.0 / 2.0, 0.052804, 0.170000, 0.370000), (-1.0 / 3.0, 0.097321, 0.400000, 1.980000),
            (1.0, 8.000000, 20.243600, 43.9336000)]


def _quintic(cos):
    """The piecewise quintic through _G_KNOTS at cos."""
    out = torch.zeros_like(cos)
    for (x0, v0, d0, s0), (x1, v1, d1, s1) in zip(_G_KNOTS, _G_KNOTS[1:]):
        h = x1 - x0
        a0, a1, a2 = v0, d0 * h, s0 * h * h / 2
        r0, r1, r2 = v1 - (a0 + a1 + a2), d1 * h - (a1 + 2 * a2), s1 * h * h - 2 * a2
        a3, a4, a5 = 10 * r0 - 4 * r1 + r2 / 2, -15 * r0 + 7 * r1 - r2, 6 * r0 - 3 * r1 + r2 / 2
        t = (cos - x0) / h
        p = a0 + t * (a1 + t * (a2 + t * (a3 + t * (a4 + t * a5))))
        out = torch.where((cos >= x0) & (cos <= x1), p, out)
    return out


def _rebo_pair(r):
    vr = (1 + 0.313460 / r) * 10953.544 * torch.exp(-4.7465391 * r)
    va = (12388.792 * torch.exp(-4.7204523 * r) + 17.567065 * torch.exp(-1.4332132 * r)
          + 30.714932 * torch.exp(-1.3826913 * r))
    return vr, va


def _brenner_pair(r, re, de, beta, s):
    vr = de / (s - 1) * torch.exp(-beta * math.sqrt(2 * s) * (r - re))
    va = de * s / (s - 1) * torch.exp(-beta * math.sqrt(2 / s) * (r - re))
    return vr, va


def _diamond_energy(case, x, nbr, back, box):
    """Energy of a diamond whose every bond is inside the cutoffs' plateau
    (four neighbours of weight 1, so the coordination corrections are 0), or
    None when a bond or a gap has left it."""
    d = x[:, None, :] - x[nbr]
    d = d - box * torch.round(d / box)
    r = d.norm(dim=2)
    if not bool((r < 1.7).all()):
        return None
    u = d / r[..., None]
    cos = (u[:, :, None, :] * u[:, None, :, :]).sum(-1)
    off = ~torch.eye(4, dtype=torch.bool)
    if case["potential"] == "rebo":
        vr, va = _rebo_pair(r)
        g = torch.where(off, _quintic(cos), torch.zeros_like(cos)).sum(2)
        b = (1 + g) ** -0.5
    else:
        if case["brenner_set"] == 1:
            vr, va = _brenner_pair(r, 1.315, 6.325, 1.5, 1.29)
            a0, c0, d0, delta = 0.011304, 19.0, 2.5, 0.80469
        else:
            vr, va = _brenner_pair(r, 1.39, 6.0, 2.1, 1.22)
            a0, c0, d0, delta = 0.00020813, 330.0, 3.5, 0.5
        g = a0 * (1 + (c0 / d0) ** 2 - c0 ** 2 / (d0 ** 2 + (1 + cos) ** 2))
        g = torch.where(off, g, torch.zeros_like(g)).sum(2)
        b = (1 + g) ** -delta
    bbar = (b + b[nbr, back]) / 2
    return ((vr - bbar * va) / 2).sum()


def exact(case, seed):
    """40 steps of a diamond from the perfect lattice are short enough to
    integrate here; the other cases' potentials (splines over connectivity and
    coordination, LJ with its bond-order switch) are too long to restate."""
    if case["use"] != "run" or case["system"] != "diamond" or case["size"] > 12:
        return None
    s = _system(case, seed)
    box = torch.tensor(s["box"], dtype=torch.float64)
    x = torch.tensor(s["pos"], dtype=torch.float64)
    v = torch.tensor(s["vel"], dtype=torch.float64)
    nbr = []
    for rows in torch.split(torch.arange(len(x)), 1024):
        d = x[rows, None, :] - x[None]
        d = (d - box * torch.round(d / box)).norm(dim=2)
        nbr.append(d.topk(5, dim=1, largest=False).indices[:, 1:])
    nbr = torch.cat(nbr)
    back = (nbr[nbr] == torch.arange(len(x))[:, None, None]).to(torch.int64).argmax(2)

    def force(x):
        x = x.detach().requires_grad_()
        e = _diamond_energy(case, x, nbr, back, box)
        if e is None:
            return None, None
        e.backward()
        return e.item(), -x.grad / _MASS_C * _EV_AMU

    dt = case["dt"]
    image = torch.zeros(x.shape, dtype=torch.int32)
    e, a = force(x)
    epot, etot = [], []
    for _ in range(case["steps"]):
        x = x + v * dt + a * dt * dt / 2
        e, a_new = force(x)
        if e is None:
            return None
        v = v + a * dt / 2 + a_new * dt / 2
        a = a_new
        shift = torch.floor(x / box)
        x = x - shift * box
        image += shift.to(torch.int32)
        epot.append(e)
        etot.append(e + 0.5 * _MASS_C * (v * v).sum().item() / _EV_AMU)
    out = {"pos": x.numpy(), "vel": v.numpy(), "image": None}
    if case["energies"]:
        out["epot"], out["etot"] = np.array(epot), np.array(etot)
    return out
