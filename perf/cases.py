"""The work a program has this library do, as cases that can be timed and compared.

Every case goes through the public Python classes over the C ABI, on inputs made from a seed. The sizes follow the
repository's own workloads (impressionfea_b200/workloads.py): the 64-case sweep's small meshes, the 31.9k-tet
upsetting drop-in, the 202k-tet closed-die gear blank, the 20 x 60 axisymmetric upsetting and the sweep's larger
2D meshes, and the learned warm start's training. Meshes are the seeded Delaunay fill; the seed also draws material
and friction (the sweep's ranges).

kind (one per path):
  spd       ISpdSolver seam: factorise a new matrix over an analysed pattern and solve, host arrays in and out;
  assembly  the element, pressure and friction terms of one Newton iteration: PrepareStep, matrix and residual;
  velocity  the whole Newton solution of one increment's velocity field, with the final evaluation;
  forge     one whole increment: remesh checks, velocity solution, contact and geometry update;
  plane     the same velocity solution in 2D (quads, band Cholesky);
  band      SymmetricBandMatrix.Factorize + Solve on a given band, host arrays in and out;
  network   the warm start's network: inference over all nodes, then a stretch of training.
"""
import math

import numpy as np
import torch

from impressionfea_b200.config import Forging2DConfig, Forging3DConfig
from impressionfea_b200.forging2d import ForgingSolver2D, band_factor_solve
from impressionfea_b200.forging3d import Forging3DSolver, GpuSpdSolver
from impressionfea_b200.meshes import gear_blank_case_3d, h_for_tets, upset_case_3d
from impressionfea_b200.warmstart import WarmStartNetwork


def listed():
    return [
        # a coarse mesh check behind the solver seam: one small factorisation after another, latency counts
        {"name": "spd_2k_tets", "kind": "spd", "tets": 2000},
        # the drop-in's factorisation, as a host that keeps the reference's stepper calls it
        {"name": "spd_30k_tets", "kind": "spd", "tets": 30000},
        # the largest systems that come through this seam
        {"name": "spd_100k_tets", "kind": "spd", "tets": 100000},
        # one Newton iteration's assembly on the closed-die blank's size
        {"name": "assembly_200k_tets", "kind": "assembly", "die": "gear", "tets": 200000},
        # a small case of the sweep, reference defaults (FP64, tolerance 1e-3)
        {"name": "velocity_5k_fp64", "kind": "velocity", "die": "flat", "tets": 5000, "fp32": False, "tol": 1e-3},
        # one whole increment of the upsetting drop-in, reference defaults
        {"name": "forge_30k_fp64", "kind": "forge", "die": "flat", "tets": 31857, "fp32": False, "tol": 1e-3},
        # the closed die at full size, single-precision factor, converged to the accuracy runs' 1e-6
        {"name": "velocity_200k_fp32", "kind": "velocity", "die": "gear", "tets": 200000, "fp32": True, "tol": 1e-6},
        # one whole closed-die increment at the size the warm start is trained on
        {"name": "forge_60k_fp32", "kind": "forge", "die": "gear", "tets": 60000, "fp32": True, "tol": 1e-6},
        # the published 2D case
        {"name": "plane_20x60", "kind": "plane", "nx": 20, "nz": 60, "axisymmetric": True},
        # a larger 2D case of the sweep
        {"name": "plane_45x131", "kind": "plane", "nx": 45, "nz": 131, "axisymmetric": True},
        # the band solver on its own, a wide ragged band
        {"name": "band_3001x141", "kind": "band", "n": 3001, "half_band": 141},
        # training the warm start between runs, and its inference over a full-size mesh's nodes
        {"name": "network_39k_nodes", "kind": "network", "nodes": 38941, "steps": 100, "batch": 8192},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spd", "assembly", "velocity", "velocity", "forge", "forge", "plane", "plane", "band", "network"])
    if kind == "spd":
        return {"kind": kind, "tets": _spread(rng, 1000, 80000)}
    if kind == "assembly":
        return {"kind": kind, "die": rng.choice(["flat", "gear"]), "tets": _spread(rng, 2000, 190000)}
    if kind in ("velocity", "forge"):
        fp32 = rng.random() < 0.5
        top = 120000 if fp32 else 60000
        return {"kind": kind, "die": rng.choice(["flat", "gear"]), "tets": _spread(rng, 3000, top), "fp32": fp32,
                "tol": 1e-6 if fp32 else 1e-3}
    if kind == "plane":
        nx = _spread(rng, 8, 44)
        return {"kind": kind, "nx": nx, "nz": int(nx * rng.uniform(1.6, 2.9)) + 1, "axisymmetric": rng.random() < 0.7}
    if kind == "band":
        return {"kind": kind, "n": _spread(rng, 300, 4000), "half_band": _spread(rng, 5, 140)}
    return {"kind": kind, "nodes": _spread(rng, 2000, 38000), "steps": rng.randint(10, 90), "batch": 128 * rng.randint(4, 64)}


# ---------------------------------------------------------------- inputs

def _solver3d(case, seed):
    """A context one increment into its run, as the host steps it: material and friction from the sweep's ranges."""
    rng = np.random.default_rng(seed)
    c, n, m, friction = rng.uniform(80, 200), rng.uniform(0, 0.2), rng.uniform(0.05, 0.25), rng.uniform(0.1, 0.6)
    tol = case.get("tol", 1e-3)
    if case.get("die", "flat") == "gear":
        height = 50.0
        h = h_for_tets(20.0, height, case["tets"])
        mesh, dies = gear_blank_case_3d(h, R=20.0, H=height, ramp=4.0, seed=seed)
        ds = mesh.gap0 / 200
    else:
        height = 45.0
        h = h_for_tets(15.0, height, case["tets"])
        mesh, dies = upset_case_3d(15.0, height, h, shut=0.6 * height, seed=seed)
        ds = 0.4 * height / 80
    cfg = Forging3DConfig(C=c, N=n, M=m, eps0=0.01, friction=friction, ram=50.0, h=h, ds=ds, size=height, tol=tol)
    s = Forging3DSolver(cfg, mesh, dies)
    if case.get("fp32"):
        s.set_scalar("factor_fp32", 1)
    s.prepare_step()
    return s


STATE = ("x", "vg", "contact", "eps", "dmg", "el_sig", "el_rate", "el_mean", "el_dev")


def _band(n, b, seed):
    """A symmetric positive definite band (row-wise, diagonal last) and a right-hand side."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    low = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64).mul_(1 / math.sqrt(b + 1))
    low = torch.tril(torch.triu(low, -b), -1)
    low.diagonal().copy_(1 + torch.rand(n, generator=g, device="cuda", dtype=torch.float64))
    full = low @ low.T
    i = torch.arange(n, device="cuda")[:, None]
    j = i + torch.arange(-b, 1, device="cuda")[None, :]
    band = torch.where(j >= 0, full[i.expand_as(j), j.clamp(min=0)], 0.0)
    rhs = torch.randn(n, generator=g, device="cuda", dtype=torch.float64)
    return band.cpu().numpy(), rhs.cpu().numpy()


def _samples(nodes, seed):
    """Network inputs and targets of the warm start's kind: 16 scaled features per node, 3 velocity changes."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((nodes, 16)).astype(np.float32)
    x[:, 8:11] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, nodes)]
    x[:, 11:13] = np.clip(np.abs(x[:, 11:13]) * 2, -1, 4)
    w = rng.standard_normal((16, 3)).astype(np.float32) / 4
    return x, (np.tanh(x @ w) + 0.05 * rng.standard_normal((nodes, 3))).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "spd":
        s = _solver3d(case, seed)
        s.assemble(1, 1)
        s.apply_bc()
        cp, ri = s.pattern()
        state["values"], state["rhs"] = s.array("val"), s.array("r")
        s.close()
        state["solver"] = GpuSpdSolver()
        state["solver"].analyze(len(cp) - 1, cp, ri)
    elif kind in ("assembly", "velocity", "forge"):
        s = state["solver"] = _solver3d(case, seed)
        if kind != "assembly":
            s.step()
            state["start"] = {a: s.array(a) for a in STATE}
            state["gap"], state["ds"] = s.scalar("gap"), s.scalar("ds_cur")
    elif kind == "plane":
        rng = np.random.default_rng(seed)
        cfg = Forging2DConfig(C=rng.uniform(80, 200), N=rng.uniform(0, 0.2), M=rng.uniform(0.05, 0.25),
                              friction=rng.uniform(0.1, 0.6), nx=case["nx"], nz=case["nz"],
                              axisymmetric=case["axisymmetric"])
        state["solver"] = ForgingSolver2D(cfg)
        state["solver"].step()
    elif kind == "band":
        state["band"], state["rhs"] = _band(case["n"], case["half_band"], seed)
    else:
        net = state["net"] = WarmStartNetwork(seed)
        state["x"], t = _samples(case["nodes"], seed)
        net.add_samples(state["x"], t)
        net.fit_normalisation()
        state["params"] = net.params()
    return state


# ---------------------------------------------------------------- one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "spd":
        s = state["solver"]
        s.factorize(state["values"])
        return {"x": s.solve(state["rhs"])}
    if kind == "assembly":
        s = state["solver"]
        s.prepare_step()
        energy, power = s.assemble(1, 1)
        scale = s.apply_bc()
        return {"energy": energy, "power": power, "max_diag": scale, "r": s.array("r")}
    if kind == "velocity":
        s = state["solver"]
        for a in ("vg", "el_sig"):
            s.set_array(a, state["start"][a])
        s.prepare_step()
        s.solve_velocity()
        power, reaction = s.final_evaluation()
        return {"power": power, "reaction": reaction, "vg": s.array("vg"), "el_rate": s.array("el_rate"),
                "el_mean": s.array("el_mean"), "release": s.array("release")}
    if kind == "forge":
        s = state["solver"]
        for a, v in state["start"].items():
            s.set_array(a, v)
        s.set_scalar("gap", state["gap"])
        s.set_scalar("ds_cur", state["ds"])
        info = s.step()
        return {"load": info["load"], "reaction": info["reaction"], "x": s.array("x"), "vg": s.array("vg"),
                "eps": s.array("eps"), "contact": s.array("contact")}
    if kind == "plane":
        s = state["solver"]
        s.prepare()
        s.solve_velocity()
        return {"v": s.array("v"), "el_rate": s.array("el_rate"), "el_sig": s.array("el_sig")}
    if kind == "band":
        low, x = band_factor_solve(state["band"], case["half_band"], state["rhs"])
        return {"l": low, "x": x}
    net = state["net"]
    net.set_params(state["params"])
    y = net.forward(state["x"])
    loss = net.train(case["steps"], case["batch"], 1e-3, 7)
    return {"prediction": y, "loss": loss, "params": net.params()}


# ---------------------------------------------------------------- the work that cannot be left out

def _mesh_counts(case):
    """Nodes, equations and stored entries of a mesh of about this many tets (quarter cylinders: 0.195 nodes a tet
    plus the surface's share, about 62 two-ring neighbours a node)."""
    ne = case["tets"]
    nn = 0.185 * ne + 1.1 * ne ** (2.0 / 3.0)
    return ne, nn, 3 * nn, 9 * 62.0 * nn


def _factor_work(ndof):
    """Entries and operations of a nested-dissection Cholesky factor on a 3D mesh of ndof equations: the usual
    4/3 and 2 powers, scaled to the 117k-equation closed-die factor (376 M entries, 2.2 TFLOP)."""
    return 376e6 * (ndof / 116823.0) ** (4.0 / 3.0), 2.2e12 * (ndof / 116823.0) ** 2


def _assembly_bytes(ne, nn, nnz):
    return ne * 192.0 + nn * 96.0 + nnz * 20.0 + 3 * nn * 9.0


def work(case):
    kind = case["kind"]
    if kind in ("spd", "assembly", "velocity", "forge"):
        ne, nn, ndof, nnz = _mesh_counts(case)
        entries, flops = _factor_work(ndof)
        if kind == "spd":
            return {"bytes": 8 * nnz + 24 * entries + 24 * ndof, "flops": flops + 4 * entries}
        if kind == "assembly":
            return {"bytes": 2 * _assembly_bytes(ne, nn, nnz), "flops": 2500.0 * ne}
        # one factorisation, and for each of about six Newton iterations an assembly and a sweep of the factor
        size = 4 if case["fp32"] else 8
        return {"bytes": 6 * (_assembly_bytes(ne, nn, nnz) + 2 * size * entries) + size * entries,
                "flops": flops + 6 * (4 * entries + 2500.0 * ne)}
    if kind in ("plane", "band"):
        if kind == "band":
            n, b, its = case["n"], case["half_band"], 1
        else:
            n, b, its = 2 * (case["nx"] + 1) * (case["nz"] + 1), 2 * min(case["nx"], case["nz"]) + 5, 6
        return {"bytes": its * 16.0 * n * (b + 1), "flops": its * (float(n) * b * (b + 1) + 4.0 * n * b)}
    weights = 16 * 128 + 2 * 128 * 128 + 128 * 3
    return {"bytes": case["nodes"] * 76.0 + case["steps"] * (case["batch"] * 76.0 + 28.0 * weights),
            "flops": 2.0 * weights * (case["nodes"] + 3 * case["steps"] * case["batch"])}


# ---------------------------------------------------------------- values in 64 bits

def exact(case, seed):
    kind = case["kind"]
    if kind == "spd":
        s = _solver3d(case, seed)
        s.assemble(1, 1)
        s.apply_bc()
        cp, ri = s.pattern()
        val, rhs = s.array("val"), s.array("r")
        s.close()
        n = len(cp) - 1
        if n > 60000:
            return None
        cols = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.from_numpy(np.diff(cp)).to("cuda", torch.int64))
        a = torch.zeros(n, n, device="cuda", dtype=torch.float64)
        a[torch.from_numpy(ri).to("cuda", torch.int64), cols] = torch.from_numpy(val).cuda()
        b = torch.from_numpy(rhs).cuda()[:, None]
        low = torch.linalg.cholesky(a)
        x = torch.cholesky_solve(b, low)
        for _ in range(2):
            x = x + torch.cholesky_solve(b - a @ x, low)
        return {"x": x[:, 0].cpu().numpy()}
    if kind == "band":
        n, b = case["n"], case["half_band"]
        band, rhs = _band(n, b, seed)
        i = torch.arange(n)[:, None]
        j = i + torch.arange(-b, 1)[None, :]
        keep = j >= 0
        a = torch.zeros(n, n, dtype=torch.float64)
        a[i.expand_as(j)[keep], j[keep]] = torch.from_numpy(band)[keep]
        a = (a + torch.tril(a, -1).T).cuda()
        low = torch.linalg.cholesky(a)
        x = torch.cholesky_solve(torch.from_numpy(rhs).cuda()[:, None], low)[:, 0]
        low = low.cpu()
        out = torch.where(keep, low[i.expand_as(j), j.clamp(min=0)], 0.0)
        return {"l": out.reshape(-1).numpy(), "x": x.cpu().numpy()}
    if kind == "network":
        # the untrained network's prediction; where a stretch of training leads has no such value
        net = WarmStartNetwork(seed)
        p = net.params().astype(np.float64)
        net.close()
        x, t = _samples(case["nodes"], seed)
        x, t = x.astype(np.float64), t.astype(np.float64)
        out, at, sizes = (x - x.mean(0)) / x.std(0), 0, [(16, 128), (128, 128), (128, 128), (128, 3)]
        for k, (a, b) in enumerate(sizes):
            w, at = p[at:at + a * b].reshape(b, a), at + a * b
            bias, at = p[at:at + b], at + b
            out = out @ w.T + bias
            if k < 3:
                out = torch.nn.functional.gelu(torch.from_numpy(out)).numpy()
        return {"prediction": out * t.std(0) + t.mean(0), "loss": None, "params": None}
    return None
