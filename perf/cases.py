"""Timed cases: the calls that programs built on this framework make, from a 192-atom force call to the
98,304-atom benchmark box.

Kinds of case (``kind``), each with the precision forms that it is used in:
  force     what an external MD driver or sampler does per step: a typed neighbour list at the new
            positions, then energies, forces and virial on it (NeighborBuilder.build, DeviceModel.evaluate)
  frames    the same for ring-polymer beads or a batch of configurations in one launch sequence
  evaluate  the reference's evaluate(): host arrays in, host arrays out
  packed    one ragged batch of the serving loop (evaluate_packed)
  nlist     the neighbour list alone, as a driver with its own force loop rebuilds it
  md        a Simulation: new positions and velocities, ten velocity-Verlet steps, the trajectory

Systems are liquid water at the density of the repository's 192-atom box (64 H2O in 12.42 A).  Models:
``water`` is the benchmark model (25-50-100 / 240^3 / axis 16), ``compact`` the shape of the reference's
training default (32-32-64 / 128^3 / axis 12) with its embedding nets tabulated.

Energies and virials are returned in single precision, the precision of the per-atom and per-pair terms
that they are sums of and the one that programs keep them in beside the forces.
"""
import functools
import math
import os
import sys
import tempfile

import numpy as np
import torch

if os.path.abspath("deepmd-jax_b200") not in sys.path:
    sys.path.insert(0, os.path.abspath("deepmd-jax_b200"))

RCUT, SKIN = 6.0, 0.3
SEL = (56, 112)          # list columns per neighbour type: the most that liquid water has, with room to spare
MODELS = {"water": dict(embed=(25, 50, 100), fit=(240, 240, 240), axis=16, grids=0),
          "compact": dict(embed=(32, 32, 64), fit=(128, 128, 128), axis=12, grids=1024)}
MASS = (15.9994, 1.0078)
MASS_UNIT = 1.036427e2   # Dalton -> eV fs^2 / A^2
KB = 8.617333e-5         # eV / K
PACK = (32, 333, 64, 100, 1025, 41, 700, 129, 57, 512, 211, 1500)  # waters of one serving batch's requests


def listed():
    return [
        # the smallest call: one 192-atom frame per step, where launches and latency are the cost
        dict(name="force192_fp32", kind="force", model="water", precision="fp32", waters=64, frames=1),
        dict(name="force192_mixed", kind="force", model="water", precision="mixed", waters=64, frames=1),
        # evaluate() as a script calls it on a handful of frames (an odd molecule count), default precision
        dict(name="evaluate8x999_fp32", kind="evaluate", model="water", precision="fp32", waters=333, frames=8),
        # the 12,288-atom box of the NVT workload, both forms
        dict(name="force12k_fp32", kind="force", model="water", precision="fp32", waters=4096, frames=1),
        dict(name="force12k_mixed", kind="force", model="water", precision="mixed", waters=4096, frames=1),
        # the 98,304-atom benchmark box, both forms
        dict(name="force98k_fp32", kind="force", model="water", precision="fp32", waters=32768, frames=1),
        dict(name="force98k_mixed", kind="force", model="water", precision="mixed", waters=32768, frames=1),
        # path-integral beads: 32 frames of 1,536 atoms in one call
        dict(name="beads32x1536_mixed", kind="force", model="water", precision="mixed", waters=512, frames=32),
        # a ragged batch as the serving loop packs it: requests of 96 to 4,500 atoms
        dict(name="packed12_mixed", kind="packed", model="water", precision="mixed", waters=1, frames=1),
        # tabulated embedding nets, what training with the default settings leaves behind
        dict(name="compact12k_fp32", kind="force", model="compact", precision="fp32", waters=4096, frames=1),
        # the neighbour list alone at the largest size
        dict(name="nlist98k", kind="nlist", model="water", precision="fp32", waters=32768, frames=1),
        # ten MD steps through Simulation, from host state to host trajectory
        dict(name="md12k_mixed", kind="md", model="water", precision="mixed", waters=4096, frames=1),
    ]


def draw(rng):
    kind = rng.choice(["force", "force", "force", "frames", "evaluate", "packed", "nlist", "md"])
    precision = rng.choice(["fp32", "mixed"])
    model = "compact" if rng.random() < 0.2 else "water"

    def logint(lo, hi):
        return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))

    frames = 1
    if kind == "force":
        waters = logint(32, 30000)
    elif kind == "frames":
        kind, waters, frames = "force", logint(64, 1200), rng.randint(2, 16)
    elif kind == "evaluate":
        waters, frames = logint(32, 1200), rng.randint(1, 12)
    elif kind == "packed":
        waters = logint(1, 4) if precision == "mixed" else 1
    elif kind == "nlist":
        waters = logint(64, 32768)
    else:
        waters = logint(80, 2000)
    return dict(kind=kind, model=model, precision=precision, waters=waters, frames=frames)


# ---------------------------------------------------------------- inputs
def _side(waters):
    return 12.42 * (waters / 64.0) ** (1.0 / 3.0)


def _water(rng, waters):
    """Positions (3 waters, 3) float64, O H H per molecule: O on sites of a jittered cubic lattice (a random choice
    of them where the number is no cube), H at the gas-phase geometry with a random orientation; types; box."""
    side = _side(waters)
    n = math.ceil(waters ** (1.0 / 3.0) - 1e-9)
    grid = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    grid = grid[np.sort(rng.permutation(len(grid))[:waters])]
    o = (grid + 0.5) * (side / n) + rng.normal(scale=0.1, size=(waters, 3))
    u = rng.normal(size=(waters, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    v = rng.normal(size=(waters, 3))
    v -= (v * u).sum(1, keepdims=True) * u
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    half = math.radians(104.52) / 2
    h1 = o + 0.9572 * (math.cos(half) * u + math.sin(half) * v)
    h2 = o + 0.9572 * (math.cos(half) * u - math.sin(half) * v)
    return np.stack([o, h1, h2], 1).reshape(-1, 3), np.tile([0, 1, 1], waters), np.full(3, side)


def _jet(layers, x):
    """Value and first two derivatives of an embedding net (tanh layers, repeat residual) at x (n,)."""
    f = [x[:, None], np.ones((len(x), 1)), np.zeros((len(x), 1))]
    for k, (w, b) in enumerate(layers):
        w = w.astype(np.float64)
        z, dz, ddz = f[0] @ w + b, f[1] @ w, f[2] @ w
        t = np.tanh(z)
        new = [t, (1 - t * t) * dz, (1 - t * t) * (ddz - 2 * t * dz * dz)]
        f = new if k == 0 else [a + np.repeat(p, a.shape[1] // p.shape[1], axis=1) for a, p in zip(new, f)]
    return f


def _table(layers, lo, hi, grids):
    """poly_coeff (grids, 6, W) of the quintics that match value, slope and curvature at both ends of each interval."""
    f, d, c = _jet(layers, np.linspace(lo, hi, grids + 1))
    h = (hi - lo) / grids
    a0, a1, a2 = f[:-1], d[:-1], c[:-1] / 2
    e0 = f[1:] - (a0 + a1 * h + a2 * h * h)
    e1 = (d[1:] - (a1 + 2 * a2 * h)) * h
    e2 = (c[1:] - 2 * a2) * h * h
    a3, a4, a5 = 10 * e0 - 4 * e1 + e2 / 2, -15 * e0 + 7 * e1 - e2, 6 * e0 - 3 * e1 + e2 / 2
    return np.stack([a5 / h ** 5, a4 / h ** 4, a3 / h ** 3, a2, a1, a0], axis=1).astype(np.float32)


@functools.lru_cache(maxsize=None)
def _model(name):
    """(params, variables) of a randomly initialised energy model in the layout of model.pkl."""
    spec = MODELS[name]
    rng = np.random.default_rng(0)

    def dense(i, o):
        return {"kernel": (rng.normal(size=(i, o)) * math.sqrt(2.0 / (i + o))).astype(np.float32),
                "bias": np.zeros(o, np.float32)}

    var, tables = {"Tbias": np.zeros(spec["embed"][-1], np.float32)}, {}
    for k in range(4):
        widths = (1,) + spec["embed"]
        net = {"Dense_%d" % i: dense(widths[i], widths[i + 1]) for i in range(3)}
        var["embedding_net_%d" % k] = net
        if spec["grids"]:
            layers = [(net["Dense_%d" % i]["kernel"], net["Dense_%d" % i]["bias"]) for i in range(3)]
            t = 0.4 / RCUT
            hi = (1 - 3 * t * t + 2 * t ** 3) / 0.4
            tables["embedding_net_%d" % k] = {"srmin": np.float32(0), "srmax": np.float32(hi),
                                              "poly_coeff": _table(layers, 0.0, float(np.float32(hi)), spec["grids"])}
    for t in range(2):
        widths = (spec["axis"] * spec["embed"][-1],) + spec["fit"] + (1,)
        net = {"Dense_%d" % i: dense(widths[i], widths[i + 1]) for i in range(4)}
        for i in (1, 2):
            net["dt%d" % i] = (0.1 + rng.normal(scale=0.001, size=widths[i + 1])).astype(np.float32)
        var["fitting_net_%d" % t] = net
    params = dict(type="energy", atomic_data_prefix=None, embed_widths=list(spec["embed"]), embedMP_widths=None,
                  fit_widths=list(spec["fit"]), axis=spec["axis"], Ebias=np.zeros(2, np.float32), rcut=RCUT,
                  use_2nd=True, use_mp=False, atomic=False, hybrid=False, nsel=None, out_norm=1.0, ntypes=2,
                  valid_types=np.arange(2), sr_mean=np.zeros(2), sr_std=np.ones(2), Nnbrs=100.0)
    variables = {"params": var}
    if tables:
        params["is_compressed"] = True
        variables["compress_var"] = tables
    return params, variables


@functools.lru_cache(maxsize=None)
def _model_file(name):
    from deepmd_jax_b200.dpmodel import DPModel
    from deepmd_jax_b200.utils import save_model
    path = os.path.join(tempfile.mkdtemp(prefix="dpcase_"), "model.pkl")
    params, variables = _model(name)
    save_model(path, DPModel(params), variables)
    return path


def _frames(case, seed):
    """Frames (F, N, 3) float64 of one system: beads and batches are displaced copies of one configuration."""
    rng = np.random.default_rng([seed, 1])
    pos, types, box = _water(rng, case["waters"])
    n = case["frames"]
    out = np.broadcast_to(pos, (n,) + pos.shape).copy()
    if n > 1:
        out += rng.normal(scale=0.05, size=out.shape)
    return out, types, box


def _velocities(seed, types):
    rng = np.random.default_rng([seed, 2])
    m = np.asarray(MASS)[types] * MASS_UNIT
    v = rng.normal(size=(len(types), 3)) * np.sqrt(KB * 300.0 / m)[:, None]
    return v - (v * m[:, None]).sum(0) / m.sum()


def _requests(case):
    return [w * case["waters"] for w in PACK]


def _request(seed, k, waters):
    return _water(np.random.default_rng([seed, 3, k]), waters)


def prepare(case, seed):
    from deepmd_jax_b200.engine import DeviceModel, NeighborBuilder, PackedBatch, sort_by_type
    kind = case["kind"]
    s = {"kind": kind, "precision": case["precision"]}
    if kind == "evaluate":
        coord, types, box = _frames(case, seed)
        return dict(s, path=_model_file(case["model"]), coord=coord, types=types, box=np.tile(box, (len(coord), 1)))
    params, variables = _model(case["model"])
    if kind == "md":
        from deepmd_jax_b200.md import Simulation
        coord, types, box = _frames(case, seed)
        vel = _velocities(seed, types)
        sim = Simulation((params, variables), box, types, MASS, "NVE", 0.5, coord[0], initial_velocity=vel,
                         report_interval=1000000, precision=case["precision"], verbose=False)
        return dict(s, sim=sim, coord=coord[0], vel=vel)
    dm = DeviceModel(params, variables)
    if kind == "packed":
        reqs = [_request(seed, k, w) for k, w in enumerate(_requests(case))]
        batch = PackedBatch([(types, 1, box) for _, types, box in reqs], 2)
        slots = np.zeros((batch.natoms, 3), np.float32)
        slots[:batch.nreal] = np.concatenate([p for p, _, _ in reqs])
        return dict(s, dm=dm, batch=batch, sel=list(SEL), pos=torch.tensor(slots, device="cuda"))
    coord, types, box = _frames(case, seed)
    f, n = coord.shape[:2]
    perm, count = sort_by_type(types, 2)
    perm = torch.tensor(perm.astype(np.int32), device="cuda")
    pos = torch.tensor(coord, dtype=torch.float32, device="cuda")
    nb = NeighborBuilder(n, f, count, SEL, box, RCUT + SKIN)
    return dict(s, dm=dm, nb=nb, pos=pos, perm=perm, count=count, sel=list(SEL),
                counts=torch.empty((f, n, 2), dtype=torch.int32, device="cuda"),
                box=torch.tensor(np.tile(box, (f, 1)), dtype=torch.float32, device="cuda"))


# ---------------------------------------------------------------- one pass
def run(s):
    if s["kind"] == "evaluate":
        from deepmd_jax_b200.train import evaluate
        r = evaluate(s["path"], s["coord"], s["box"], s["types"], batch_size=8, precision=s["precision"])
        return {"energy": r["energy"].astype(np.float32), "force": r["force"]}
    if s["kind"] == "md":
        sim = s["sim"]
        sim.setPosition(s["coord"])
        sim.setVelocity(s["vel"])
        t = sim.run(10)
        return {"position": t["position"].astype(np.float32), "velocity": t["velocity"].astype(np.float32)}
    if s["kind"] == "packed":
        from deepmd_jax_b200.engine import evaluate_packed
        out = evaluate_packed(s["dm"], s["batch"], s["pos"], s["sel"], RCUT, precision=s["precision"], atom_energy=True)
        return {"energy": out["energy"].float(), "force": out["force"], "virial": out["virial"].float(),
                "atom_energy": out["atom_energy"], "nbrs": out["nbrs"], "status": out["status"]}
    if s["kind"] == "nlist":
        nbrs, status = s["nb"].build(s["pos"], perm=s["perm"], counts=s["counts"])
        return {"nbrs": nbrs, "counts": s["counts"], "status": status}
    nbrs, status = s["nb"].build(s["pos"], perm=s["perm"])
    out = s["dm"].evaluate(s["pos"], s["box"], nbrs, s["count"], s["sel"], perm=s["perm"], precision=s["precision"],
                           atom_energy=True, status=status)
    return {"nbrs": nbrs, "energy": out["energy"].float(), "force": out["force"], "virial": out["virial"].float(),
            "atom_energy": out["atom_energy"], "status": out["status"]}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    spec = MODELS[case["model"]]
    if case["kind"] == "packed":
        atoms = 3 * sum(_requests(case))
    else:
        atoms = 3 * case["waters"] * case["frames"]
    density = 192 / 12.42 ** 3
    listed_rows = density * 4 / 3 * math.pi * (RCUT + SKIN) ** 3   # list entries per atom
    rows = density * 4 / 3 * math.pi * RCUT ** 3                   # pairs within the cutoff per atom
    e, a, f = spec["embed"], spec["axis"], spec["fit"]
    net = (10 * e[2] if spec["grids"] else 2 * (e[0] + e[0] * e[1] + e[1] * e[2])) + 20 * e[2]
    fit = 2 * (a * e[2] * f[0] + f[0] * f[1] + f[1] * f[2] + f[2]) + 20 * a * e[2]
    flops = 2.0 * (rows * net + fit)        # forward and adjoint
    weights = 4.0 * (2 * (a * e[2] * f[0] + f[0] * f[1] + f[1] * f[2])
                     + 4 * (6 * spec["grids"] * e[2] if spec["grids"] else e[0] * e[1] + e[1] * e[2]))
    if case["kind"] == "nlist":
        return {"bytes": atoms * (12 + 4 * listed_rows + 8), "flops": atoms * listed_rows * 8.0}
    steps = 11 if case["kind"] == "md" else 1
    per_atom = {"evaluate": 24 + 12, "md": 48 + 48 * 10}.get(case["kind"], 12 + 4 * listed_rows + 12 + 4)
    return {"bytes": atoms * per_atom + weights, "flops": steps * atoms * flops}


# ---------------------------------------------------------------- 64-bit values
def _net64(spec, variables, k, st):
    def t(x):
        return torch.as_tensor(np.asarray(x), dtype=torch.float64, device=st.device)
    if spec["grids"]:
        tab = variables["compress_var"]["embedding_net_%d" % k]
        delta = (float(tab["srmax"]) - float(tab["srmin"])) / spec["grids"]
        x = st - float(tab["srmin"])
        idx = (x / delta).to(torch.int64)
        x0 = (x - idx * delta)[:, None]
        c = t(tab["poly_coeff"])[idx.clamp(0, spec["grids"] - 1)]
        h = c[:, 0]
        for i in range(1, 6):
            h = h * x0 + c[:, i]
        return h
    h = st[:, None]
    for i in range(3):
        d = variables["params"]["embedding_net_%d" % k]["Dense_%d" % i]
        z = torch.tanh(h @ t(d["kernel"]) + t(d["bias"]))
        h = z if i == 0 else z + h.repeat_interleave(z.shape[1] // h.shape[1], dim=1)
    return h


def _fit64(variables, t, g):
    net = variables["params"]["fitting_net_%d" % t]
    for i in range(4):
        w, b = (torch.as_tensor(net["Dense_%d" % i][n], dtype=torch.float64, device=g.device) for n in ("kernel", "bias"))
        z = g @ w + b
        if i == 3:
            return z[:, 0]
        z = torch.tanh(z)
        g = z if i == 0 else z * torch.as_tensor(net["dt%d" % i], dtype=torch.float64, device=g.device) + g


def _eval64(name, pos, box, types):
    """Energy, atom energies, forces and virial of one frame: pos (N, 3) float64, box (3,), every periodic image."""
    spec, (params, variables) = MODELS[name], _model(name)
    dev, n, a = pos.device, len(pos), spec["axis"]
    r2 = math.sqrt(2.0)
    reach = [int(math.floor(RCUT / float(b) + 0.5)) for b in box]
    shifts = torch.tensor([[i, j, k] for i in range(-reach[0], reach[0] + 1) for j in range(-reach[1], reach[1] + 1)
                           for k in range(-reach[2], reach[2] + 1)], dtype=torch.float64, device=dev) * box
    e_atom = torch.zeros(n, dtype=torch.float64, device=dev)
    force, virial = torch.zeros_like(pos), torch.zeros(3, 3, dtype=torch.float64, device=dev)
    for t in range(2):
        centres = torch.nonzero(types == t)[:, 0]
        for ci in centres.split(1024):
            pair, x = [], []
            for sh in shifts:
                d = pos[None] - pos[ci][:, None]
                d = d - box * torch.round(d / box) + sh
                q = (d * d).sum(-1)
                hit = torch.nonzero((q < RCUT * RCUT) & (q > 1e-20))
                pair.append(hit)
                x.append(d[hit[:, 0], hit[:, 1]])
                del d, q
            pair, x = torch.cat(pair), torch.cat(x).requires_grad_(True)
            i, j = pair[:, 0], pair[:, 1]
            r = x.norm(dim=1)
            u = r / RCUT
            s = (1 - 3 * u ** 2 + 2 * u ** 3) / r
            xh = x / r[:, None]
            env = torch.cat([torch.ones_like(s)[:, None], math.sqrt(3.0) * xh, 3 * (xh * xh - 1.0 / 3),
                             3 * r2 * xh * xh.roll(1, 1)], 1) * s[:, None]
            desc = torch.zeros(len(ci), 10, spec["embed"][2], dtype=torch.float64, device=dev)
            for tj in range(2):
                m = types[j] == tj
                h = _net64(spec, variables, 2 * t + tj, s[m])
                desc = desc.index_add(0, i[m], env[m][:, :, None] * h[:, None, :])
            desc = desc / params["Nnbrs"]
            t3, t6 = desc[:, 1:4], desc[:, 4:]
            y = t3[:, :, a:2 * a]
            g2 = torch.cat([y * y, r2 * y * y.roll(1, 1)], 1) + t6[:, :, a:2 * a]
            g = (torch.einsum("nca,ncw->naw", desc[:, :4, :a], desc[:, :4]) + torch.einsum("nca,ncw->naw", g2, t6))
            e = _fit64(variables, t, g.reshape(len(ci), -1))
            dx, = torch.autograd.grad(e.sum(), x)
            e_atom[ci] = e.detach()
            force.index_add_(0, ci[i], dx)
            force.index_add_(0, j, -dx)
            virial -= x.detach().T @ dx
    return e_atom.sum(), e_atom, force, virial


def exact(case, seed):
    kind, name = case["kind"], case["model"]
    if kind == "nlist":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def f32(a):  # inputs reach the device in single precision
        return torch.tensor(np.asarray(a, np.float32), device=dev).double()

    if kind == "packed":
        reqs = [_request(seed, k, w) for k, w in enumerate(_requests(case))]
        got = [_eval64(name, f32(p), f32(b), torch.tensor(t, device=dev)) for p, t, b in reqs]
        natoms = sum((-(-w // 8) + -(-2 * w // 8)) * 8 for w in _requests(case))
        pad = natoms - sum(len(g[1]) for g in got)
        return {"energy": torch.stack([g[0] for g in got]), "virial": torch.stack([g[3].reshape(9) for g in got]),
                "force": torch.cat([g[2] for g in got] + [torch.zeros(pad, 3, dtype=torch.float64, device=dev)]),
                "atom_energy": None, "nbrs": None, "status": None}
    coord, types, box = _frames(case, seed)
    types, box = torch.tensor(types, device=dev), f32(box)
    if kind == "md":
        x, v = f32(coord[0]), torch.tensor(_velocities(seed, types.cpu().numpy()), device=dev)
        m = torch.tensor(np.asarray(MASS)[types.cpu().numpy()] * MASS_UNIT, device=dev)[:, None]
        px, pv = [x], [v]
        f = _eval64(name, x, box, types)[2]
        for _ in range(10):
            v = v + 0.25 * f / m
            x = x + 0.5 * v
            f = _eval64(name, x, box, types)[2]
            v = v + 0.25 * f / m
            px.append(x)
            pv.append(v)
        return {"position": torch.stack(px), "velocity": torch.stack(pv)}
    got = [_eval64(name, f32(c), box, types) for c in coord]
    energy, force = torch.stack([g[0] for g in got]), torch.stack([g[2] for g in got])
    if kind == "evaluate":
        return {"energy": energy, "force": force}
    return {"nbrs": None, "energy": energy, "force": force, "virial": torch.stack([g[3].reshape(9) for g in got]),
            "atom_energy": torch.stack([g[1] for g in got]), "status": None}
