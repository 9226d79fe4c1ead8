"""The work that the framework is measured on: one dict of plain values per case.

Every case is a block that a differentiable flow-map program runs through the public entry points: a march of the
flow maps over a reinit interval, the advections, the BFECC pullbacks, the adjoint's sources, the projections (plain
and with an obstacle), the control forces, a kernel's backward pass, and two whole gradients.  Sizes are those of
the repository's configurations (128^3 shape transition, 128^2 .. 384^2 vortex batch, 3000 Gaussians) and odd,
ragged ones beside them.

``exact`` restates each block in plain torch in 64 bits (None for the whole gradients).
"""
from __future__ import annotations

import importlib
import itertools
import math

import numpy as np
import torch

PKG = "differentiable-flowmap_b200"
K = importlib.import_module(PKG + ".kernels")
A = importlib.import_module(PKG + ".autograd")
MG = importlib.import_module(PKG + ".mgpcg")
C = importlib.import_module(PKG + ".configs")
SIM = importlib.import_module(PKG + ".simulator")
VORTEX = importlib.import_module(PKG + ".vortex")

DT = {"f32": torch.float32, "f64": torch.float64}


# ------------------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the in-interval replay of a reinit: the maps psi, T marched back through one interval of midpoint velocities
        {"name": "flow_map_3d128", "kind": "flow_map", "n0": 128, "n1": 128, "n2": 128, "rk": 4, "marches": 8,
         "dtype": "f32"},
        # the same on a small ragged 2D grid (dx not a power of two), where launches count
        {"name": "flow_map_2d_ragged", "kind": "flow_map", "n0": 250, "n1": 333, "n2": 0, "rk": 2, "marches": 12,
         "dtype": "f32"},
        # the adjoint step's advections: two velocities and two scalars back along one midpoint velocity
        {"name": "advect_pair_3d128", "kind": "advect", "n0": 128, "n1": 128, "n2": 128, "rk": 4, "pair": True,
         "dtype": "f32"},
        # the reinit's pullbacks (BFECC of the velocity and of a scalar) in the FP64 runs that errors are stated against
        {"name": "bfecc_3d_ragged_f64", "kind": "bfecc", "n0": 90, "n1": 77, "n2": 101, "dtype": "f64"},
        # the adjoint step's sources and their accumulation through the maps
        {"name": "adjoint_sources_3d128", "kind": "sources", "n0": 128, "n1": 128, "n2": 128, "dtype": "f32"},
        # a pressure projection of the 3D shape transition, the mixed-precision solver settings
        {"name": "project_3d128", "kind": "project", "n0": 128, "n1": 128, "n2": 128, "levels": 5, "pre_post": 3,
         "bottom": 50, "mode": 0, "rel_tol": 3e-7, "bf16": True, "dtype": "f32"},
        # a pressure projection of the 2D vortex optimisation
        {"name": "project_2d256", "kind": "project", "n0": 256, "n1": 256, "n2": 0, "levels": 5, "pre_post": 2,
         "bottom": 20, "mode": 1, "rel_tol": 1e-10, "bf16": False, "dtype": "f32"},
        # the same around a leaf-shaped obstacle
        {"name": "project_obstacle_2d256", "kind": "obstacle", "n0": 256, "levels": 5, "rel_tol": 1e-10,
         "angle": 0.6, "dtype": "f32"},
        # Gaussian control forces of the 3D optimisation: the force field, and the sums over its adjoint
        {"name": "control_forces_3d128", "kind": "forces", "n0": 128, "n1": 128, "n2": 128, "count": 3000,
         "dtype": "f32"},
        # a kernel composed with torch: the RK4 self-advection and its backward pass
        {"name": "advect_backward_3d64", "kind": "backward", "n0": 64, "n1": 64, "n2": 64, "rk": 4, "dtype": "f32"},
        # a whole 2D vortex gradient (forward, adjoint, d loss / d theta), replayed from its CUDA graph
        {"name": "vortex_gradient_2d256", "kind": "vortex", "n0": 256, "steps": 20, "reinit": 10, "dtype": "f32"},
        # a whole 3D gradient in the checkpointed form: one full reinit interval and a partial one
        {"name": "gradient_3d128", "kind": "gradient", "n0": 128, "steps": 12, "reinit": 8, "form": "checkpointed",
         "dtype": "f32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flow_map", "advect", "bfecc", "sources", "project", "obstacle", "forces", "backward",
                       "vortex", "gradient"])
    c = {"kind": kind, "dtype": "f32"}
    if kind in ("flow_map", "advect", "bfecc", "sources", "forces"):
        if rng.random() < 0.6:
            c.update(n0=_log_int(rng, 24, 140), n1=_log_int(rng, 24, 140), n2=_log_int(rng, 24, 140))
        else:
            c.update(n0=_log_int(rng, 48, 768), n1=_log_int(rng, 48, 768), n2=0)
        if kind != "forces" and rng.random() < 0.25:
            c["dtype"] = "f64"
    if kind == "flow_map":
        c.update(rk=rng.choice([2, 4]), marches=rng.randint(1, 10))
    elif kind == "advect":
        c.update(rk=rng.choice([2, 4]), pair=rng.random() < 0.5)
    elif kind == "forces":
        c["count"] = _log_int(rng, 16, 3000)
    elif kind == "project":
        if rng.random() < 0.5:
            lv = rng.randint(3, 5)
            m = 1 << (lv - 1)
            n = [m * max(2, rng.randint(24 // m, 144 // m)) for _ in range(3)]
            c.update(n0=n[0], n1=n[1], n2=n[2], levels=lv, pre_post=rng.choice([2, 3]), bottom=50, mode=0,
                     rel_tol=rng.choice([3e-6, 1e-6, 3e-7]), bf16=rng.random() < 0.5)
        else:
            lv = rng.randint(4, 5)
            m = 1 << (lv - 1)
            n = [m * rng.randint(64 // m, 512 // m) for _ in range(2)]
            c.update(n0=n[0], n1=n[1], n2=0, levels=lv, pre_post=2, bottom=20, mode=1,
                     rel_tol=rng.choice([1e-6, 1e-8, 1e-10]), bf16=False)
        if not c["bf16"] and rng.random() < 0.2:
            c["dtype"] = "f64"
    elif kind == "obstacle":
        c.update(n0=rng.choice([128, 192, 256, 320, 384]), levels=4, rel_tol=rng.choice([1e-6, 1e-8, 1e-10]),
                 angle=round(rng.uniform(0.0, 1.5), 3))
    elif kind == "backward":
        c.update(n0=_log_int(rng, 16, 72), n1=_log_int(rng, 16, 72), n2=_log_int(rng, 16, 72), rk=rng.choice([2, 4]))
    elif kind == "vortex":
        c.update(n0=rng.choice([128, 192, 256, 384]), steps=rng.randint(4, 16), reinit=rng.choice([5, 10]))
    elif kind == "gradient":
        c.update(n0=rng.choice([32, 64, 128]), steps=rng.randint(2, 9), reinit=rng.choice([4, 8]),
                 form=rng.choice(["plain", "mixed", "checkpointed"]))
    return c


# ----------------------------------------------------------------------------------------------------------- inputs
def _res(c):
    return (c["n0"], c["n1"]) if c["n2"] == 0 else (c["n0"], c["n1"], c["n2"])


def _faces(res):
    return [tuple(n + (a == f) for a, n in enumerate(res)) for f in range(len(res))]


def _field(g, shape, rms, dtype):
    """A random field with a k^(-11/6) amplitude spectrum (that of a turbulent velocity) plus 2 % white noise."""
    k = torch.meshgrid(*[torch.fft.fftfreq(n, d=1.0 / n, device="cuda") for n in shape], indexing="ij")
    k2 = sum(x * x for x in k)
    amp = torch.where(k2 > 0, k2.clamp(min=1.0) ** (-11.0 / 12.0 - 0.25 * (len(shape) - 2)), torch.zeros_like(k2))
    f = torch.fft.ifftn(torch.fft.fftn(torch.randn(shape, generator=g, device="cuda")) * amp).real
    f = f / f.square().mean().sqrt() + 0.02 * torch.randn(shape, generator=g, device="cuda")
    return (rms * f).to(dtype).contiguous()


def _mac(g, res, rms, dtype):
    return [_field(g, s, rms, dtype) for s in _faces(res)]


def _nodes(res, face, dx, dtype):
    """Positions of the nodes of a face grid (face -1: cell centres), (dim, *grid)."""
    axes = [(torch.arange(n + (a == face), device="cuda", dtype=torch.float64) + (0.0 if a == face else 0.5)) * dx
            for a, n in enumerate(res)]
    return torch.stack(torch.meshgrid(*axes, indexing="ij")).to(dtype).contiguous()


def _maps(g, res, dx, dtype):
    """Flow maps as an interval leaves them: identity plus about a cell of displacement, Jacobian rows near e_c."""
    dim = len(res)
    psi, T = [], []
    for c, s in enumerate(_faces(res)):
        p, t = _nodes(res, c, dx, dtype), torch.zeros((dim,) + s, dtype=dtype, device="cuda")
        t[c] = 1
        for a in range(dim):
            p[a] += _field(g, s, 1.5 * dx, dtype)
            t[a] += _field(g, s, 0.1, dtype)
        psi.append(p)
        T.append(t)
    pc = _nodes(res, -1, dx, dtype)
    for a in range(dim):
        pc[a] += _field(g, res, 1.5 * dx, dtype)
    return psi, T, pc


def _ball(res, center, radius, dx):
    x = _nodes(res, -1, dx, torch.float64)
    r = sum((x[a] - center[a]) ** 2 for a in range(len(res))).sqrt()
    return (0.5 * (1.0 - torch.tanh((r - radius) / dx))).float()


def _split(g, res, std):
    """Cell-centred white noise split to the faces (the optimisation's starting velocity)."""
    out = []
    for c in range(len(res)):
        v = torch.randn(res, generator=g, device="cuda") * std
        n = v.shape[c]
        out.append((0.5 * (torch.cat([v.narrow(c, 0, 1), v], c) + torch.cat([v, v.narrow(c, n - 1, 1)], c))).contiguous())
    return out


def prepare(case, seed):
    c, kind, dtype = case, case["kind"], DT[case["dtype"]]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if kind == "obstacle":
        res = (c["n0"], c["n0"])
        mask = torch.as_tensor(C.leaf_mask(c["n0"], angle=c["angle"]))
        solver = MG.MGPCG_2_solid(boundary_mask=mask, N=res, dtype=dtype, levels=c["levels"], abs_tol=0.0,
                                  rel_tol=c["rel_tol"], check_every=0)
        return {"c": c, "solver": solver, "u": _mac(g, res, 0.3, dtype)}
    if kind == "vortex":
        cfg = C.vortex2d_config(res=c["n0"], steps=c["steps"], reinit_every=c["reinit"], rel_tol=1e-10)
        problem = VORTEX.VortexProblem(SIM.LFM_Diff_Simulator(config=cfg))
        theta = C.vortex2d_theta(seed)
        target = problem.final_vorticity(C.vortex2d_theta(seed + 1))
        problem.capture(theta, target)
        return {"c": c, "problem": problem, "theta": theta, "target": target}
    if kind == "gradient":
        n = c["n0"]
        mixed = c["form"] != "plain"
        cfg = C.shape3d_config(res=n, steps=c["steps"], reinit_every=c["reinit"], backward_u=not mixed,
                               rel_tol=3e-7 if mixed else 3e-6, coarse_bf16=mixed,
                               store_dtype=torch.bfloat16 if c["form"] == "mixed" else None)
        if mixed:
            cfg.solver.pre_post = 3
        if c["form"] == "checkpointed":
            cfg.recompute = cfg.ckpt_delta = True
        rng = np.random.default_rng(seed)
        rho = torch.maximum(*[_ball((n,) * 3, rng.uniform(0.3, 0.7, 3), rng.uniform(0.08, 0.14), 1.0 / n)
                              for _ in range(2)])
        return {"c": c, "sim": SIM.LFM_Diff_Simulator(config=cfg), "u0": _split(g, (n,) * 3, 0.01),
                "rho0": _ball((n,) * 3, (0.5,) * 3, 0.15, 1.0 / n), "rho": rho}
    res = _res(c)
    s = {"c": c, "grid": K.GridSpec(res), "dx": 1.0 / res[0], "dt": 0.0085 * 128 / res[0]}
    if kind == "flow_map":
        s["u"] = [_mac(g, res, 0.3, dtype) for _ in range(c["marches"])]
        s["psi"], s["T"] = ([torch.empty((len(res),) + f, dtype=dtype, device="cuda") for f in _faces(res)]
                            for _ in range(2))
        s["psi_c"] = torch.empty((len(res),) + res, dtype=dtype, device="cuda")
    elif kind == "advect":
        s["u"] = _mac(g, res, 0.3, dtype)
        s["fields"] = [_mac(g, res, 0.3, dtype) for _ in range(1 + c["pair"])]
        s["scalars"] = [_field(g, res, 1.0, dtype) for _ in range(1 + c["pair"])]
        s["fields_out"] = [[torch.empty_like(x) for x in f] for f in s["fields"]]
        s["scalars_out"] = [torch.empty_like(x) for x in s["scalars"]]
    elif kind == "bfecc":
        s["u"], s["s"] = _mac(g, res, 0.3, dtype), _field(g, res, 1.0, dtype)
        s["maps"], s["back"] = _maps(g, res, s["dx"], dtype), _maps(g, res, s["dx"], dtype)
        s["u1"], s["u2"], s["u3"] = ([torch.empty_like(x) for x in s["u"]] for _ in range(3))
        s["s1"], s["s2"], s["s3"] = (torch.empty_like(s["s"]) for _ in range(3))
    elif kind == "sources":
        s["u"], s["w"], s["init"], s["Hp"], s["Hpp"] = (_mac(g, res, 0.3, dtype) for _ in range(5))
        s["s"], s["lam"] = _field(g, res, 1.0, dtype), _field(g, res, 1.0, dtype)
        s["psi"], s["T"], _ = _maps(g, res, s["dx"], dtype)
        s["src"], s["src_s"] = ([torch.empty_like(x) for x in s["u"]] for _ in range(2))
        s["acc"], s["hp"], s["hpp"] = ([torch.empty_like(x) for x in s["u"]] for _ in range(3))
    elif kind == "project":
        s["solver"] = MG.MGPCG(res, dtype, levels=c["levels"], pre_post=c["pre_post"], bottom=c["bottom"],
                               bottom_mode=c["mode"], abs_tol=0.0, rel_tol=c["rel_tol"], check_every=0,
                               eps=1e-12 if dtype == torch.float32 else 0.0, coarse_bf16=c["bf16"])
        s["u"] = _mac(g, res, 0.3, dtype)
    elif kind == "forces":
        n, d = c["count"], len(res)
        ext = torch.tensor([r / res[0] for r in res], device="cuda")
        s["center"] = (torch.rand(n, d, generator=g, device="cuda") * ext).contiguous()
        s["center"] = s["center"].to(dtype)
        ks = torch.tensor([1, 1, 1, 1, 2, 3, 4, 5, 6, 7, 8, 9], device="cuda")  # radii in cells, as the optimiser draws them
        s["inv_r"] = (ks[torch.randint(12, (n,), generator=g, device="cuda")] * s["dx"]).square().reciprocal().to(dtype)
        s["strength"] = (0.02 * torch.randn(n, d, generator=g, device="cuda")).to(dtype)
        s["f"] = [torch.empty(f, dtype=dtype, device="cuda") for f in _faces(res)]
        s["adj"] = _mac(g, res, 0.3, dtype)
    elif kind == "backward":
        s["u"] = [x.requires_grad_() for x in _mac(g, res, 0.3, dtype)]
        s["lam"] = _mac(g, res, 1.0, dtype)
    return s


# -------------------------------------------------------------------------------------------------------------- run
def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind in ("project", "obstacle"):
        return A.project(s["solver"], s["u"])
    if kind == "vortex":
        loss, dtheta = s["problem"].graph_gradient(s["theta"])
        # (the parameters' gradient in the run's type, as the optimiser's update takes it; so too the forces' below)
        return {"loss": loss, "dtheta": torch.from_numpy(dtheta).to(DT[c["dtype"]]), "adj_u": s["problem"].sim.adj_u}
    if kind == "gradient":
        loss, grads = s["sim"].gradient(s["u0"], s["rho0"], s["rho"])
        return {"loss": loss, "grads": grads}
    g, dx, dt = s["grid"], s["dx"], s["dt"]
    if kind == "flow_map":
        K.reset_to_identity(g, dx, s["psi_c"], s["psi"], s["T"])
        for u in s["u"]:
            K.march_map(g, c["rk"], dx, dt, s["psi_c"], s["psi"], s["T"], u)
        return {"psi_c": s["psi_c"], "psi": s["psi"], "T": s["T"]}
    if kind == "advect":
        f, o, a, b = s["fields"], s["fields_out"], s["scalars"], s["scalars_out"]
        if c["pair"]:
            K.advect_u_grid_pair(g, c["rk"], dx, -dt, s["u"], f[0], o[0], f[1], o[1])
            K.advect_scalar_grid_pair(g, c["rk"], dx, -dt, s["u"], a[0], b[0], a[1], b[1])
        else:
            K.advect_u_grid(g, c["rk"], dx, dt, s["u"], f[0], o[0])
            K.advect_scalar_grid(g, c["rk"], dx, dt, s["u"], a[0], b[0])
        return {"fields": o, "scalars": b}
    if kind == "bfecc":
        (psi, T, psi_c), (phi, F, phi_c) = s["maps"], s["back"]
        K.pullback_u(g, dx, s["u"], s["u1"], T, psi)
        K.pullback_u(g, dx, s["u1"], s["u2"], F, phi, alpha=0.5, beta=-1.0, base=s["u"])
        K.pullback_u(g, dx, s["u2"], s["u3"], T, psi, alpha=-1.0, beta=-1.0, base=s["u1"])
        K.pullback_scalar(g, dx, s["s"], s["s1"], psi_c)
        K.pullback_scalar(g, dx, s["s1"], s["s2"], phi_c, alpha=0.5, beta=-1.0, base=s["s"])
        K.pullback_scalar(g, dx, s["s2"], s["s3"], psi_c, alpha=-1.0, beta=-1.0, base=s["s1"])
        return {"u": s["u3"], "s": s["s3"]}
    if kind == "sources":
        K.nabla_u_w(g, dx, s["u"], s["w"], s["src"])
        K.nabla_scalar_adjoint(g, dx, s["s"], s["lam"], s["src_s"])
        for to, of in (("acc", "init"), ("hp", "Hp"), ("hpp", "Hpp")):  # a simulator's running sums, as each step finds them
            for x, y in zip(s[to], s[of]):
                x.copy_(y)
        K.accumulate_init_pair(g, dx, -2 * dt, s["src"], s["acc"], s["T"], s["psi"], s["src_s"], -dt, s["hp"],
                               s["hpp"], 3)
        return {"src": s["src"], "src_s": s["src_s"], "acc": s["acc"], "hp": s["hp"]}
    if kind == "forces":
        K.gaussian_force(g, dx, s["center"], s["inv_r"], s["strength"], s["f"])
        sums = K.gaussian_force_grad(g, dx, s["center"], s["inv_r"], s["strength"], s["adj"])
        return {"f": s["f"], "sums": [x.to(s["adj"][0].dtype) for x in sums]}
    out = A.advect_u_grid(s["u"], s["u"], dx, dt, c["rk"])
    return {"out": [x.detach() for x in out], "grads": torch.autograd.grad(out, s["u"], s["lam"])}


# ------------------------------------------------------------------------------------------------------------- work
def work(case):
    c, kind = case, case["kind"]
    b = 4 if c["dtype"] == "f32" else 8
    if kind in ("obstacle", "vortex"):
        res = (c["n0"],) * 2
    elif kind == "gradient":
        res = (c["n0"],) * 3
    else:
        res = _res(c)
    dim, n = len(res), math.prod(res)
    nf = sum(math.prod(f) for f in _faces(res))
    mac = dim * 3 ** dim * 2        # flops of one velocity sample (a multiply-add per tap)
    rk = c.get("rk", 2)
    if kind == "flow_map":
        # psi, T are written; each march reads its velocity; a sample of the gradient is three contractions
        per = nf * rk * mac * 2 + n * rk * mac
        return {"bytes": b * (dim * 2 * nf + dim * n + c["marches"] * nf), "flops": c["marches"] * per}
    if kind == "advect":
        m = 1 + c["pair"]
        return {"bytes": b * (nf + 2 * m * (nf + n)), "flops": (nf + n) * (rk * mac + m * 2 * 3 ** dim)}
    if kind == "bfecc":
        return {"bytes": b * (2 * (2 * dim * nf + dim * n) + 2 * (nf + n)), "flops": 3 * (nf * (mac + 2 * dim) + n * 2 * 3 ** dim)}
    if kind == "sources":
        taps = 4 if dim == 3 else 5
        return {"bytes": b * (2 * nf + 2 * n + 2 * nf + 2 * dim * nf + 6 * nf),
                "flops": nf * dim * taps * dim * 4 + nf * dim * 8 * 2 + 2 * nf * mac}
    if kind in ("project", "obstacle"):
        # the velocity in and out; one V-cycle's sweeps, residual and transfers per cell, and a PCG update
        return {"bytes": b * 2 * nf, "flops": n * (2 * dim + 2) * 8}
    if kind == "forces":
        # faces in the support (radius sqrt(5) k cells) of an average Gaussian
        support = math.pi * (4 / 3 * 5 ** 1.5 * 169.1 if dim == 3 else 5 * 24.1)
        return {"bytes": b * 2 * nf, "flops": 2 * dim * c["count"] * min(support, n) * 6}
    if kind == "backward":
        return {"bytes": b * 4 * nf, "flops": nf * (rk * mac * 4 + 4 * 3 ** dim)}
    steps = c["steps"]  # a forward and an adjoint step: a march, two advections and two projections each way
    per = b * (30 * nf) if kind == "gradient" else b * (24 * nf)
    return {"bytes": steps * per, "flops": steps * (6 * nf * rk * mac + 4 * n * (2 * dim + 2) * 8)}


# ------------------------------------------------------------------------------------------------------------ exact
def _axis(x, dx, stag, n, order=2):
    """Taps and weights (and their derivatives) of a B-spline along one axis at positions x."""
    length = n + 1 if stag else n
    s = (x / dx - (0.0 if stag else 0.5)).clamp(min=None, max=length - 2 - 1e-6).clamp(min=1.0)
    lo = {2: -1, 3: -2, 4: -3}[order]
    iu = torch.floor(s.detach())
    taps, w, d = [], [], []
    for t in range({2: 4, 3: 6, 4: 8}[order]):
        y = s - (iu + lo + t)
        a, sg = y.abs(), torch.where(y < 0, -1.0, 1.0)
        z = torch.zeros_like(a)
        if order == 2:
            v = torch.where(a < 0.5, 0.75 - a * a, torch.where(a < 1.5, 0.5 * (1.5 - a) ** 2, z))
            e = torch.where(a < 0.5, -2 * a, torch.where(a < 1.5, a - 1.5, z))
        elif order == 3:
            v = torch.where(a < 1, 0.5 * a ** 3 - a * a + 2 / 3, torch.where(a < 2, (2 - a) ** 3 / 6, z))
            e = torch.where(a < 1, 1.5 * a * a - 2 * a, torch.where(a < 2, -0.5 * (2 - a) ** 2, z))
        else:
            v = torch.where(a < 0.5, 115 / 192 - 5 * a * a / 8 + a ** 4 / 4, torch.where(
                a < 1.5, 55 / 96 + 5 * a / 24 - 5 * a * a / 4 + 5 * a ** 3 / 6 - a ** 4 / 6,
                torch.where(a < 2.5, (2.5 - a) ** 4 / 24, z)))
            e = torch.where(a < 0.5, -1.25 * a + a ** 3, torch.where(
                a < 1.5, 5 / 24 - 2.5 * a + 2.5 * a * a - 2 / 3 * a ** 3,
                torch.where(a < 2.5, -((2.5 - a) ** 3) / 6, z)))
        taps.append((iu + lo + t).long().clamp(0, length - 1))
        w.append(v)
        d.append(sg * e / dx)
    return taps, w, d


def _sample(f, p, dx, res, stag, order=2, grad=False):
    """Value (and gradient) of a field at positions p (list of dim tensors); stag: its staggered axis or -1."""
    dim = len(res)
    ax = [_axis(p[a], dx, a == stag, res[a], order) for a in range(dim)]
    flat, stride = f.reshape(-1), [math.prod(f.shape[a + 1:]) for a in range(dim)]
    v, gr = 0, [0] * dim
    for t in itertools.product(*[range(len(x[0])) for x in ax]):
        q = flat[sum(ax[a][0][t[a]] * stride[a] for a in range(dim))]
        v = v + q * math.prod([ax[a][1][t[a]] for a in range(dim)])
        for b in range(dim if grad else 0):
            gr[b] = gr[b] + q * math.prod([ax[a][2 if a == b else 1][t[a]] for a in range(dim)])
    return (v, gr) if grad else v


def _velocity(u, p, dx, res):
    return [_sample(u[c], p, dx, res, c) for c in range(len(res))]


def _foot(u, X, dx, dt, res, rk):
    d = range(len(res))
    v1 = _velocity(u, X, dx, res)
    v2 = _velocity(u, [X[a] - 0.5 * dt * v1[a] for a in d], dx, res)
    if rk == 2:
        return [X[a] - dt * v2[a] for a in d]
    v3 = _velocity(u, [X[a] - 0.5 * dt * v2[a] for a in d], dx, res)
    v4 = _velocity(u, [X[a] - dt * v3[a] for a in d], dx, res)
    return [X[a] - dt * (v1[a] + 2 * v2[a] + 2 * v3[a] + v4[a]) / 6 for a in d]


def _march(u, psi, T, dx, dt, res, rk):
    """One Runge-Kutta march of positions and Jacobian rows through u, time step -dt."""
    d, h = range(len(res)), -dt

    def stage(p, t):
        if t is None:
            return _velocity(u, p, dx, res), None
        s = [_sample(u[c], p, dx, res, c, grad=True) for c in d]
        return [x[0] for x in s], [sum(s[c][1][b] * t[b] for b in d) for c in d]

    def at(f, k, hh):
        return None if f is None else [f[a] + hh * k[a] for a in d]

    k1, d1 = stage(psi, T)
    k2, d2 = stage(at(psi, k1, h / 2), at(T, d1, h / 2))
    if rk == 2:
        return at(psi, k2, h), at(T, d2, h)
    k3, d3 = stage(at(psi, k2, h / 2), at(T, d2, h / 2))
    k4, d4 = stage(at(psi, k3, h), at(T, d3, h))

    def end(f, x1, x2, x3, x4):
        return None if f is None else [f[a] + h * (x1[a] + 2 * x2[a] + 2 * x3[a] + x4[a]) / 6 for a in d]

    return end(psi, k1, k2, k3, k4), end(T, d1, d2, d3, d4)


def _poisson(u, fluid=None):
    """u minus the gradient of the pressure that makes it free of divergence (walls, and faces of solid cells, closed)."""
    dim, res = len(u), tuple(u[0].shape[a] - (a == 0) for a in range(len(u)))
    u = [x.clone() for x in u]

    def close():
        for c in range(dim):
            u[c].select(c, 0).zero_()
            u[c].select(c, res[c]).zero_()
            if fluid is not None:
                u[c].narrow(c, 1, res[c] - 1).mul_(fluid.narrow(c, 1, res[c] - 1) * fluid.narrow(c, 0, res[c] - 1))

    close()
    b = -sum(torch.diff(u[c], dim=c) for c in range(dim))
    if fluid is None:
        lam, mats = 0, []
        for c, n in enumerate(res):
            i = torch.arange(n, device="cuda", dtype=torch.float64)
            m = torch.cos(math.pi * i[:, None] * (i[None] + 0.5) / n) * math.sqrt(2.0 / n)
            m[0] /= math.sqrt(2.0)
            mats.append(m)
            lam = lam + (2 - 2 * torch.cos(math.pi * i / n)).reshape([-1 if a == c else 1 for a in range(dim)])
        x = b
        for c in range(dim):
            x = torch.movedim(torch.tensordot(mats[c], x, dims=([1], [c])), 0, c)
        lam[(0,) * dim] = 1.0
        x = x / lam
        x[(0,) * dim] = 0.0  # the pressure's mean
        for c in range(dim):
            x = torch.movedim(torch.tensordot(mats[c], x, dims=([0], [c])), 0, c)
    else:
        def op(x):
            y = torch.zeros_like(x)
            for c in range(dim):
                d = torch.diff(x, dim=c) * fluid.narrow(c, 1, res[c] - 1) * fluid.narrow(c, 0, res[c] - 1)
                y.narrow(c, 0, res[c] - 1).sub_(d)
                y.narrow(c, 1, res[c] - 1).add_(d)
            return y

        x, r = torch.zeros_like(b), b * fluid
        p, rr = r.clone(), (r * r).sum()
        first = float(rr)
        for it in range(12000):
            q = op(p)
            a = rr / (p * q).sum()
            x += a * p
            r -= a * q
            new = (r * r).sum()
            if it % 100 == 0 and float(new) <= 1e-26 * first:
                break
            p = r + (new / rr) * p
            rr = new
    for c in range(dim):
        u[c].narrow(c, 1, res[c] - 1).sub_(torch.diff(x, dim=c))
    close()
    return u


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("vortex", "gradient"):
        return None  # a whole simulation
    s = prepare(c, seed)
    d64 = lambda v: [d64(x) for x in v] if isinstance(v, (list, tuple)) else v.detach().double()  # noqa: E731
    if kind == "project":
        return _poisson(d64(s["u"]))
    if kind == "obstacle":
        return _poisson(d64(s["u"]), 1.0 - (s["solver"].mask > 0).double())
    res, dx, dt = _res(c), s["dx"], s["dt"]
    dim, rk = len(res), c.get("rk")
    u = d64(s["u"]) if "u" in s else None
    if kind == "flow_map":
        psi, T = [], []
        for f in range(-1, dim):
            p = list(_nodes(res, f, dx, torch.float64))
            t = None if f < 0 else [torch.full_like(p[0], float(a == f)) for a in range(dim)]
            for v in u:
                p, t = _march(v, p, t, dx, dt, res, rk)
            psi.append(torch.stack(p))
            T.append(None if t is None else torch.stack(t))
        return {"psi_c": psi[0], "psi": psi[1:], "T": T[1:]}
    if kind == "advect":
        sg = -dt if c["pair"] else dt
        feet = [_foot(u, list(_nodes(res, f, dx, torch.float64)), dx, sg, res, rk) for f in range(-1, dim)]
        return {"fields": [[_sample(x[a], feet[a + 1], dx, res, a) for a in range(dim)] for x in d64(s["fields"])],
                "scalars": [_sample(x, feet[0], dx, res, -1) for x in d64(s["scalars"])]}
    if kind == "bfecc":
        (psi, T, pc), (phi, F, hc) = d64(s["maps"]), d64(s["back"])

        def pull(v, M, m):
            at = [_velocity(v, list(m[a]), dx, res) for a in range(dim)]
            return [sum(M[a][b] * at[a][b] for b in range(dim)) for a in range(dim)]

        u1 = pull(u, T, psi)
        u2 = [0.5 * (x - y) for x, y in zip(pull(u1, F, phi), u)]
        s0 = d64(s["s"])
        s1 = _sample(s0, list(pc), dx, res, -1)
        s2 = 0.5 * (_sample(s1, list(hc), dx, res, -1) - s0)
        return {"u": [y - x for x, y in zip(pull(u2, T, psi), u1)], "s": s1 - _sample(s2, list(pc), dx, res, -1)}
    if kind == "sources":
        w, lam, sc = d64(s["w"]), d64(s["lam"]), d64(s["s"])
        order = 3 if dim == 3 else 4

        def fixed(f, stag, face, deriv, order):  # the separable stencil at the nodes of a face grid, axis by axis
            for a in range(dim):
                x = (torch.arange(res[a] + (a == face), device="cuda", dtype=torch.float64) + (0.0 if a == face else 0.5)) * dx
                taps, wt, dw = _axis(x, dx, a == stag, res[a], order)
                sh = [-1 if b == a else 1 for b in range(dim)]
                f = sum(f.index_select(a, t) * (e if a == deriv else v).reshape(sh) for t, v, e in zip(taps, wt, dw))
            return f

        src = [sum(fixed(u[a], a, f, f, order) * fixed(w[a], a, f, None, order) for a in range(dim)) for f in range(dim)]
        src_s = [fixed(sc, -1, f, f, 3) * fixed(lam, -1, f, None, 3) for f in range(dim)]
        psi, T = d64(s["psi"]), d64(s["T"])
        acc, hp = [], []
        for f in range(dim):
            at = [sum(T[f][b] * v for b, v in enumerate(_velocity(x, list(psi[f]), dx, res))) for x in (src, src_s)]
            hp.append(at[0])
            acc.append(s["init"][f].double() + (23 * at[0] - 16 * s["Hp"][f].double() + 5 * s["Hpp"][f].double()) / 12 * (-2 * dt) - dt * at[1])
        return {"src": src, "src_s": src_s, "acc": acc, "hp": hp}
    if kind == "forces":
        return None  # the support's sharp edge falls on other nodes in 64 bits
    # backward: torch's own derivative of the 64-bit advection, one component at a time
    u = [x.requires_grad_() for x in u]
    outs, grads = [], [0] * dim
    for f in range(dim):
        o = _sample(u[f], _foot(u, list(_nodes(res, f, dx, torch.float64)), dx, dt, res, rk), dx, res, f)
        gr = torch.autograd.grad(o, u, s["lam"][f].double())
        grads = [a + b for a, b in zip(grads, gr)]
        outs.append(o.detach())
    return {"out": outs, "grads": grads}
