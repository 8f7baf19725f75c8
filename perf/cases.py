"""The work that users of phipict_b200 have it do, as measurable cases.

Five kinds, each called through the package's public entry points:

- ``step``: one ``single_step()`` of a running simulation (momentum predictor, two pressure
  correctors and, with a magnetic field, the potential step and the Lorentz force);
- ``run``: a new simulation on a prepared domain, started from a given velocity and run for a
  few steps;
- ``batch``: the same as ``step`` of a ``DomainBatch`` of simulations of different sizes, Hartmann and
  Reynolds numbers and time steps;
- ``gradient``: a checkpointed rollout and its reverse pass (``adjoint.rollout``);
- ``assembly``: the backend protocol's assembly calls of one step without the solves, as a
  driver that brings its own solver calls them.

Precisions: ``f32`` and ``f64`` are the plain paths (CG and BiCGStab in the domain's type),
``mixed`` is float32 Krylov iterations with the multigrid preconditioner inside float64
refinement. Grids are rectilinear: a periodic channel between walls, a lid-driven cavity, a
duct of blocks connected along x, graded towards its walls.

:func:`exact` restates the discretisation in float64 with plain torch on whole arrays and
solves its systems with a Jacobi-preconditioned CG and a BiCGStab of its own.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

# One step of the C1 channel, the cavity of the validation runs at an odd size, the duct of the
# default benchmark on the plain and on the mixed path, ragged and single-block ducts, the
# heterogeneous batches and the differentiable duct.
_LISTED = [
    # the smallest simulation that is run in earnest: the 2D Hartmann channel, float32, 200
    # steps in a row; launches and synchronisations count
    dict(name="channel_64x32_f32", kind="step", shape="channel", nx=64, ny=32, nz=1, blocks=1, precision="f32", dt=1e-3,
         ha=10.0, re=100.0, rtol=1e-8, guesses="", warm=1),
    # lid-driven cavity without a magnetic field, odd sizes, with a transported passive scalar:
    # the plain float64 path of small 2D validation runs
    dict(name="cavity_129x121_f64", kind="step", shape="cavity", nx=129, ny=121, nz=1, blocks=1, precision="f64", dt=2e-3,
         ha=0.0, re=1000.0, rtol=1e-10, guesses="", warm=0),
    # the benchmark's duct on the plain float64 path, the path every result is checked against
    dict(name="duct_3x64x48x48_f64", kind="step", shape="duct", nx=64, ny=48, nz=48, blocks=3, precision="f64", dt=0.01,
         ha=100.0, re=1000.0, rtol=1e-10, guesses="", warm=1),
    # the benchmark's duct as the benchmark runs it: mixed precision, multigrid, projected
    # initial guesses from the last 12 results; twelve steps from the start, since with such
    # guesses the work of a step depends on how far the run has come
    dict(name="duct_3x64x48x48_mixed", kind="run", shape="duct", nx=64, ny=48, nz=48, blocks=3, precision="mixed", dt=0.01,
         ha=100.0, re=1000.0, rtol=1e-10, guesses="projection:12", steps=12),
    # a ragged duct (odd cells along every axis, so no row is aligned and the coarse levels end
    # in single-cell aggregates) with phiPICT's own initial guesses
    dict(name="duct_2x37x45x41_mixed", kind="step", shape="duct", nx=37, ny=45, nz=41, blocks=2, precision="mixed", dt=0.01,
         ha=30.0, re=1000.0, rtol=1e-10, guesses="", warm=1),
    # the largest single simulation of the serving mix
    dict(name="duct_128x128x128_mixed", kind="step", shape="duct", nx=128, ny=128, nz=128, blocks=1, precision="mixed",
         dt=0.005, ha=20.0, re=1000.0, rtol=1e-8, guesses="", warm=1),
    # a grid whose solver vectors are far larger than L2, plain float64
    dict(name="duct_160x144x144_f64", kind="step", shape="duct", nx=160, ny=144, nz=144, blocks=1, precision="f64", dt=0.005,
         ha=20.0, re=1000.0, rtol=1e-8, guesses="", warm=0),
    # 64 channels and cavities of 32^2 to 256^2 cells advanced together (parameter sweeps)
    dict(name="batch_64_2d_mixed", kind="batch", dims=2, instances=64, low=32, high=256, mix=0, precision="mixed", rtol=1e-8,
         warm=1),
    # a serving batch of ducts of 32^3 to 128^3 cells
    dict(name="batch_6_3d_mixed", kind="batch", dims=3, instances=6, low=32, high=112, mix=3, precision="mixed", rtol=1e-8,
         warm=1),
    # gradient of a loss on the final velocity through a rollout with respect to the inflow
    # profile and the Stuart number, forward and reverse pass
    dict(name="gradient_2x48x96x96", kind="gradient", nx=48, ny=96, nz=96, blocks=2, steps=2, dt=0.01, ha=10.0, re=1000.0,
         rtol=1e-12),
    # assembly of one step on grids far larger than L2, float64 and (2D, odd) float32
    dict(name="assembly_192x192x192_f64", kind="assembly", dims=3, nx=192, ny=192, nz=192, precision="f64"),
    dict(name="assembly_1999x1501_f32", kind="assembly", dims=2, nx=1999, ny=1501, nz=1, precision="f32"),
]


def listed():
    return [dict(c) for c in _LISTED]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: every kind with sizes over its range, even and odd."""
    kind = rng.choice(["channel", "cavity", "duct_f64", "duct_mixed", "duct_mixed", "batch2", "batch3", "gradient", "assembly"])
    if kind == "channel":
        return dict(kind="step", shape="channel", nx=_log(rng, 32, 256), ny=_log(rng, 16, 200), nz=1, blocks=1,
                    precision=rng.choice(["f32", "f64"]), dt=1e-3, ha=round(rng.uniform(1, 20), 2), re=100.0, rtol=1e-8,
                    guesses="", warm=1)
    if kind == "cavity":
        return dict(kind="step", shape="cavity", nx=_log(rng, 33, 300), ny=_log(rng, 33, 300), nz=1, blocks=1, precision="f64",
                    dt=2e-3, ha=0.0, re=float(rng.randint(100, 2000)), rtol=1e-10, guesses="", warm=0)
    if kind in ("duct_f64", "duct_mixed"):
        blocks = rng.randint(1, 3)
        top = 120 if kind == "duct_f64" else 110
        c = dict(kind="step", shape="duct", nx=max(12, _log(rng, 24, top) // blocks), ny=_log(rng, 20, top),
                 nz=_log(rng, 20, top), blocks=blocks, precision=kind.split("_")[1], dt=0.005,
                 ha=round(math.exp(rng.uniform(math.log(2), math.log(100))), 2), re=1000.0, rtol=rng.choice([1e-8, 1e-10]),
                 guesses="", warm=2)
        if kind == "duct_mixed" and rng.random() < 0.4:
            del c["warm"]
            c.update(kind="run", guesses="projection:12", steps=rng.randint(4, 12))
        return c
    if kind == "batch2":
        return dict(kind="batch", dims=2, instances=rng.randint(6, 60), low=rng.randint(24, 48), high=rng.randint(64, 256),
                    mix=rng.randint(1, 10 ** 6), precision="mixed", rtol=1e-8, warm=1)
    if kind == "batch3":
        return dict(kind="batch", dims=3, instances=rng.randint(2, 6), low=rng.randint(20, 32), high=rng.randint(40, 96),
                    mix=rng.randint(1, 10 ** 6), precision="mixed", rtol=1e-8, warm=1)
    if kind == "gradient":
        return dict(kind="gradient", nx=_log(rng, 16, 48), ny=_log(rng, 24, 72), nz=_log(rng, 24, 72), blocks=2, steps=2, dt=0.01,
                    ha=10.0, re=1000.0, rtol=1e-12)
    if rng.random() < 0.5:
        return dict(kind="assembly", dims=2, nx=_log(rng, 100, 2000), ny=_log(rng, 100, 2000), nz=1,
                    precision=rng.choice(["f32", "f64"]))
    return dict(kind="assembly", dims=3, nx=_log(rng, 32, 190), ny=_log(rng, 32, 190), nz=_log(rng, 32, 190),
                precision=rng.choice(["f32", "f64"]))


# --- grids and inputs, shared by the product and the exact path -------------------------------
def _tanh_nodes(n, beta=2.0):
    xi = np.linspace(-1.0, 1.0, n + 1)
    return np.tanh(beta * xi) / np.tanh(beta)


def _nodes(shape, nx, ny, nz, blocks):
    """Node coordinates per axis (x over all blocks)."""
    if shape == "channel":
        return [np.linspace(0.0, 4.0, nx + 1), np.linspace(-1.0, 1.0, ny + 1)]
    if shape == "cavity":
        return [np.linspace(0.0, 1.0, nx + 1), np.linspace(0.0, 1.0, ny + 1)]
    if shape == "square":  # 2D assembly: a channel graded towards its walls
        return [np.linspace(0.0, 4.0, nx + 1), _tanh_nodes(ny)]
    return [np.linspace(0.0, 2.0 * blocks, nx * blocks + 1), _tanh_nodes(ny), _tanh_nodes(nz)]


def _noise(gen, shape, device):
    return torch.randn(shape, generator=gen, dtype=torch.float64, device=device)


def _inputs(shape, nx, ny, nz, blocks, seed, device):
    """Initial velocity [D, z, y, x] over the whole domain, the inflow profile [3, z, y] of a
    duct and the scalar field of a cavity, float64."""
    gen = torch.Generator(device=device).manual_seed(seed)
    d = 3 if shape == "duct" else 2
    n = (nz, ny, nx * blocks) if d == 3 else (1, ny, nx)
    u = (1e-2 if shape == "duct" else 1e-3) * _noise(gen, (d,) + n, device)
    if shape != "cavity":
        u[0] += 1.0
    inflow = scalar = None
    if shape == "duct":
        inflow = torch.zeros(3, nz, ny, dtype=torch.float64, device=device)
        inflow[0] = 1.0 + 1e-2 * _noise(gen, (nz, ny), device)
    if shape == "cavity":
        scalar = torch.rand(n, generator=gen, dtype=torch.float64, device=device)
    return u, inflow, scalar


def _vertices(axes, dtype, device):
    t = [torch.as_tensor(a, dtype=torch.float64, device=device) for a in axes]
    if len(t) == 2:
        Y, X = torch.meshgrid(t[1], t[0], indexing="ij")
        v = torch.stack([X, Y])
    else:
        Z, Y, X = torch.meshgrid(t[2], t[1], t[0], indexing="ij")
        v = torch.stack([X, Y, Z])
    return v.unsqueeze(0).to(dtype).contiguous()


def _build(shape, nx, ny, nz, blocks, re, dtype, seed, device):
    """A prepared domain and its initial state."""
    import phipict_b200 as pb

    axes = _nodes(shape, nx, ny, nz, blocks)
    u, inflow, scalar = _inputs(shape, nx, ny, nz, blocks, seed, device)
    d = len(axes)
    dom = pb.Domain(d, torch.tensor([1.0 / re]), name=shape, device=device, dtype=dtype)
    bl = []
    for i in range(blocks):
        xs = axes[0][i * nx:(i + 1) * nx + 1]
        bl.append(dom.CreateBlock(vertexCoordinates=_vertices([xs] + axes[1:], dtype, device), name=f"b{i}"))
    if shape == "duct":
        for i in range(blocks - 1):
            bl[i].ConnectBlock("+x", bl[i + 1], "-x", "-y", "-z")
        face = inflow.to(dtype).reshape(1, 3, nz, ny, 1)
        bl[0].CloseBoundary("-x", face)
        bl[-1].CloseBoundary("+x", face.clone())
        bl[-1].getBoundary("+x").setPotentialBC(pb.PotentialBC.OPEN)
        for b in bl:
            for f in ("-y", "+y", "-z", "+z"):
                b.CloseBoundary(f)
    elif shape == "cavity":
        for f in ("-x", "+x", "-y"):
            bl[0].CloseBoundary(f)
        lid = torch.zeros(1, 2, 1, nx, dtype=dtype, device=device)
        lid[0, 0] = 1.0
        bl[0].CloseBoundary("+y", lid)
        bl[0].setPassiveScalar(scalar.to(dtype).reshape(1, 1, ny, nx))
    else:
        bl[0].CloseBoundary("-y")
        bl[0].CloseBoundary("+y")
        bl[0].MakePeriodic("x")
    for i, b in enumerate(bl):
        b.velocity.copy_(u[..., i * nx:(i + 1) * nx].reshape(b.velocity.shape).to(dtype))
    dom.PrepareSolve()
    return dom


def _reset_source(domain, **kw):
    # the Lorentz force is added onto the velocity source: a run without another forcing
    # clears it every step
    src = getattr(domain, "_src", None)
    if src is not None:
        src.zero_()


def _simulation(dom, case, dt, stuart):
    import phipict_b200 as pb

    tol = pb.SolverTolerance(rtol=case["rtol"])
    mixed = case["precision"] == "mixed"
    kw = dict(non_orthogonal=False, advection_tol=tol, pressure_tol=tol, mixed_precision=mixed, pressure_use_amg=mixed)
    if case.get("guesses"):
        kw["extrapolate_guesses"] = case["guesses"]
    if stuart is None:
        sim = pb.Simulation(dom, 1e-3 if isinstance(dt, torch.Tensor) else dt, **kw)
    else:
        hooks = pb.Hooks().append(pb.Hook.PRE_VELOCITY_SETUP, _reset_source)
        sim = pb.MHDSimulation(dom, 1e-3 if isinstance(dt, torch.Tensor) else dt, stuart,
                               torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64), potential_tol=tol,
                               potential_use_preconditioner=mixed, hooks=hooks, **kw)
    if isinstance(dt, torch.Tensor):
        sim.time_step = dt
    return sim


def _dtype(case):
    return torch.float32 if case.get("precision") == "f32" else torch.float64


def _members(case):
    """The instances of a batch: (shape, nx, ny, nz, re, stuart, dt)."""
    r = random.Random(case["mix"])
    sides = [s for s in (32, 48, 64, 96, 128, 192, 256) if case["low"] <= s <= case["high"]] or [case["low"], case["high"]]
    out = []
    for _ in range(case["instances"]):
        if case["dims"] == 2:
            side = r.choice(sides)
            shape = r.choice(["channel", "cavity"])
            ha, re = 10 ** (3 * r.random()), 100 + 1900 * r.random()
            n = ha * ha / re
            out.append((shape, side, side, 1, re, n, min(1e-3, 0.5 / n)))
        else:
            side = r.randint(case["low"], case["high"])
            ha = 10 ** (3 * r.random())
            n = ha * ha / 1000.0
            out.append(("duct", side, side, side, 1000.0, n, min(0.01, 0.5 / n)))
    return out


# --- the measured path --------------------------------------------------------------------------
def prepare(case, seed):
    import phipict_b200 as pb

    device = torch.device("cuda")
    k = case["kind"]
    if k == "step":
        dom = _build(case["shape"], case["nx"], case["ny"], case["nz"], case["blocks"], case["re"], _dtype(case), seed, device)
        stuart = None if case["shape"] == "cavity" else torch.tensor(case["ha"] ** 2 / case["re"], dtype=torch.float64)
        sim = _simulation(dom, case, case["dt"], stuart)
        for _ in range(case["warm"]):
            if not sim.single_step():
                raise RuntimeError(f"warm-up step failed: {sim.last_error}")
        return dict(case=case, dom=dom, sim=sim, scalar=case["shape"] == "cavity")
    if k == "run":
        dom = _build(case["shape"], case["nx"], case["ny"], case["nz"], case["blocks"], case["re"], _dtype(case), seed, device)
        return dict(case=case, dom=dom, initial=[b.velocity.clone() for b in dom.getBlocks()], phi=torch.zeros_like(dom.pressureResult),
                    stuart=torch.tensor(case["ha"] ** 2 / case["re"], dtype=torch.float64))
    if k == "batch":
        mem = _members(case)
        doms = [_build(s, nx, ny, nz, 1, re, torch.float64, seed * 1000 + e, device) for e, (s, nx, ny, nz, re, _, _) in enumerate(mem)]
        batch = pb.DomainBatch(doms)
        sim = _simulation(batch, case, torch.tensor([m[6] for m in mem], dtype=torch.float64),
                          torch.tensor([m[5] for m in mem], dtype=torch.float64))
        for _ in range(case["warm"]):
            if not sim.single_step():
                raise RuntimeError(f"warm-up step failed: {sim.last_error}")
        return dict(case=case, dom=batch, sim=sim, scalar=False)
    if k == "gradient":
        from phipict_b200.adjoint import AdjointMHD

        dom = _build("duct", case["nx"], case["ny"], case["nz"], case["blocks"], case["re"], torch.float64, seed, device)
        b = dom.getBlocks()
        model = AdjointMHD(dom, case["dt"], torch.tensor([case["ha"] ** 2 / case["re"]]),
                           torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64), steps=case["steps"],
                           faces=[(b[0], "-x"), (b[-1], "+x")], checkpoint_every=10, tol=case["rtol"], mixed_precision=True)
        n = dom.getTotalSize()
        initial = [torch.cat([blk.velocity.reshape(3, -1) for blk in b], dim=1).reshape(-1).clone(),
                   torch.zeros(n, dtype=torch.float64, device=device), torch.zeros(3 * n, dtype=torch.float64, device=device)]
        return dict(case=case, model=model, initial=initial, profile=b[0].getBoundary("-x").velocity.detach().clone(),
                    stuart=torch.tensor([case["ha"] ** 2 / case["re"]], dtype=torch.float64),
                    weight=_loss_weight(case, seed, device))
    shape = "duct" if case["dims"] == 3 else "square"
    dom = _build(shape, case["nx"], case["ny"], case["nz"], 1, 1000.0, _dtype(case), seed, device)
    f = _assembly_fields(case, seed, device)
    dt = _dtype(case)
    dom.SetupEpotOnDomain()
    for b in dom.getBlocks():
        b.setVelocitySource(f["src"].to(dt).reshape(b.velocity.shape))
        b.setPressure(f["p"].to(dt).reshape(b.pressure.shape))
    return dict(case=case, dom=dom, ts=torch.tensor([1e-3], dtype=torch.float64), phi=f["phi"].to(dt).reshape(-1),
                uxb=f["uxb"].to(dt).reshape(-1))


def _loss_weight(case, seed, device):
    gen = torch.Generator(device=device).manual_seed(seed + 77)
    n = case["nx"] * case["blocks"] * case["ny"] * case["nz"]
    return torch.randn(3 * n, generator=gen, dtype=torch.float64, device=device)


def _assembly_fields(case, seed, device):
    """Source, pressure, potential and u x e_b of an assembly case: smooth fields with noise."""
    gen = torch.Generator(device=device).manual_seed(seed + 5)
    d = case["dims"]
    n = (case["nz"], case["ny"], case["nx"])
    x = torch.linspace(0, 6.0, case["nx"], dtype=torch.float64, device=device)
    y = torch.linspace(0, 3.0, case["ny"], dtype=torch.float64, device=device).view(-1, 1)

    def smooth(shape):
        return torch.sin(x) * torch.cos(y) + 0.1 * _noise(gen, shape, device)

    return dict(src=smooth((d,) + n), p=smooth(n), phi=smooth(n), uxb=smooth((3,) + n))


def run(state):
    case = state["case"]
    k = case["kind"]
    if k in ("step", "batch"):
        dom, sim = state["dom"], state["sim"]
        if not sim.single_step():
            raise RuntimeError(f"step failed: {sim.last_error}")
        out = {"u": dom.velocityResult, "p": dom.pressureResult}
        if state["scalar"]:
            out["scalar"] = dom.scalarResult
        else:
            out["phi"] = dom.epotResult
        return out
    if k == "run":
        from phipict_b200 import _C

        dom = state["dom"]
        for b, u in zip(dom.getBlocks(), state["initial"]):
            b.setVelocity(u)
        _C.CopyVelocityResultFromBlocks(dom)
        sim = _simulation(dom, case, case["dt"], state["stuart"])
        dom.setEpotResult(state["phi"])
        if not sim.run(case["steps"]):
            raise RuntimeError(f"step failed: {sim.last_error}")
        return {"u": dom.velocityResult, "p": dom.pressureResult, "phi": dom.epotResult}
    if k == "gradient":
        from phipict_b200.adjoint import rollout

        prof = state["profile"].clone().requires_grad_(True)
        stuart = state["stuart"].clone().requires_grad_(True)
        u = rollout(state["model"], prof, stuart, initial=[t.clone() for t in state["initial"]])
        loss = (u.reshape(-1) * state["weight"]).sum()
        loss.backward()
        return {"u": u.detach(), "profile_grad": prof.grad, "stuart_grad": stuart.grad}
    from phipict_b200 import _C

    dom, ts = state["dom"], state["ts"]
    d = case["dims"]
    _C.CopyVelocityResultFromBlocks(dom)
    _C.SetupAdvectionMatrix(dom, ts)
    _C.SetupAdvectionVelocity(dom, ts)
    _C.SetupPressureCorrection(dom, ts)
    _C.CorrectVelocity(dom, ts, version=1)
    n = dom.getTotalSize()
    rhs = _C.ComputeEpotRHS(dom, state["uxb"][: d * n])
    J = _C.ComputeCurrentDensityFaceBased(dom, state["phi"], state["uxb"])
    return {"C": dom._stencil("C"), "A": dom.A, "rhs": dom.velocityRHS, "P": dom._stencil("P"), "hbya": dom.pressureRHS,
            "div": dom.pressureRHSdiv, "u": dom.velocityResult, "epot_rhs": rhs, "J": J}


def work(case):
    """Inputs read once and outputs written once; operations of one application of every
    kernel and of every system's matrix."""
    k = case["kind"]

    def step(cells, d, s):
        stencil = 2 * d + 1
        # transforms, velocity in; velocity, pressure and potential out; one matrix of each
        # of the three systems formed
        return cells * (2 * d * d + 1 + 2 * d + 2 + 3 * stencil) * s, cells * (40 * d + 2 * stencil * (d + 2))

    if k == "step":
        d = 3 if case["shape"] == "duct" else 2
        b, f = step(case["nx"] * case["ny"] * case["nz"] * case["blocks"], d, 4 if case["precision"] == "f32" else 8)
    elif k == "run":
        b, f = step(case["nx"] * case["ny"] * case["nz"] * case["blocks"] * case["steps"], 3, 8)
    elif k == "batch":
        b, f = step(sum(m[1] * m[2] * m[3] for m in _members(case)), case["dims"], 8)
    elif k == "gradient":
        b, f = step(case["nx"] * case["blocks"] * case["ny"] * case["nz"] * case["steps"], 3, 8)
        b, f = 3 * b, 3 * f  # the steps, their recomputation and their reverse
    else:
        d, s = case["dims"], 4 if case["precision"] == "f32" else 8
        cells = case["nx"] * case["ny"] * case["nz"]
        # transforms, u (read and copied), source, p, phi, u x e_b in; C, A, right-hand side, P,
        # HbyA, divergence, u, potential right-hand side, J out
        b = cells * s * (2 * d * d + 1 + 2 * d + d + 2 + 3 + (2 * d + 1) + 1 + d + (2 * d + 1) + d + 1 + d + 1 + 3)
        f = cells * (60 * d + 30)
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    """Measured against exact(): a solve to the relative residual rtol leaves up to 63 rtol in
    the pressure (6.3e-7 at 1e-8 on a long channel), the gradients 1.7e-10; the float32
    channel's pressure is limited by its float32 residual times the condition number, which
    grows with the square of the cells per side (2.1e-4 at 64x32); the float32 divergence
    cancels to 1.1e-4, the float64 one to 2e-13 on small grids."""
    k = case["kind"]
    if k == "assembly":
        return {"rel": 5e-4} if case["precision"] == "f32" else {"rel": 1e-11}
    if k == "gradient":
        return {"rel": 1e-9}
    if case["precision"] == "f32":
        return {"rel": min(0.02, 1e-3 * max(1.0, (max(case["nx"], case["ny"]) / 64) ** 2)), "max": 0.5}
    return {"rel": 250 * case["rtol"]}


# --- float64 restatement ------------------------------------------------------------------------
class _Solve(torch.autograd.Function):
    """x of A x = b for a stencil (diagonal and one coefficient array per face), with the
    gradients of the solution in b and in the coefficients."""

    @staticmethod
    def forward(ctx, grid, kind, b, *coef):
        x = grid.krylov(kind, coef, b)
        ctx.grid, ctx.kind = grid, kind
        ctx.save_for_backward(x, *coef)
        return x

    @staticmethod
    def backward(ctx, g):
        x, *coef = ctx.saved_tensors
        grid = ctx.grid
        if ctx.kind == "cg":
            lam = grid.krylov("cg", coef, grid.center(g))
        else:
            # row i of A^T takes from face f the coefficient that its neighbour has back to it
            t = [coef[0]] + [grid.nb(coef[1 + (f ^ 1)], f) for f in range(2 * grid.d)]
            lam = grid.krylov("bicg", t, g)
        parts = [-(lam * x)] + [-(lam * grid.nb(x, f)) for f in range(2 * grid.d)]
        if ctx.kind != "cg":
            parts = [p.reshape((-1, grid.d) + p.shape[1:]).sum(1) for p in parts]
        return (None, None, lam, *parts)


class _Grid:
    """A rectilinear box of cells, arrays [batch, z, y, x]; faces -x +x -y +y -z +z are
    periodic or prescribed (velocity per face, insulating unless open)."""

    def __init__(self, axes, periodic_x, face_velocity, open_faces, dt, nu, device):
        self.d = d = len(axes)
        self.h, self.periodic_x, self.open = [], periodic_x, open_faces
        self.dt = torch.as_tensor(dt, dtype=torch.float64, device=device).view(-1, 1, 1, 1)
        self.nu = torch.as_tensor(nu, dtype=torch.float64, device=device).view(-1, 1, 1, 1)
        n = [len(a) - 1 for a in axes]
        for a in range(d):
            shape = [1, 1, 1, 1]
            shape[3 - a] = n[a]
            self.h.append(torch.as_tensor(np.diff(axes[a]), dtype=torch.float64, device=device).view(shape))
        full = (1, n[2] if d > 2 else 1, n[1], n[0])
        det = torch.ones(full, dtype=torch.float64, device=device)
        for h in self.h:
            det = det * h
        self.det = det
        self.alpha = [det / (h * h) for h in self.h]
        self.mask = []
        for f in range(2 * d):
            m = torch.ones(full, dtype=torch.float64, device=device)
            if not (periodic_x and f < 2):
                m.narrow(3 - (f >> 1), n[f >> 1] - 1 if f & 1 else 0, 1).zero_()
            self.mask.append(m)
        self.ub = face_velocity  # face -> [d components], each broadcasting against [batch, z, y, x]

    def nb(self, x, f):
        return torch.roll(x, -1 if f & 1 else 1, dims=3 - (f >> 1))

    def bound(self, f, k):
        v = self.ub.get(f)
        return 0.0 if v is None else v[k]

    def fluxes(self, v):
        out = []
        for f in range(2 * self.d):
            a = f >> 1
            area = self.det / self.h[a]
            c = area * v[a]
            out.append(self.mask[f] * 0.5 * (c + self.nb(c, f)) + (1 - self.mask[f]) * area * self.bound(f, a))
        return out

    def momentum(self, u):
        """Diagonal and face coefficients of the advection-diffusion matrix."""
        diag = self.det / self.dt
        off = []
        for f, fl in enumerate(self.fluxes(u)):
            a, m = f >> 1, self.mask[f]
            half = 0.5 * (1.0 if f & 1 else -1.0) * fl
            coeff = 0.5 * (self.alpha[a] + self.nb(self.alpha[a], f)) * self.nu
            off.append(m * (half - coeff) / self.det)
            diag = diag + m * (half + coeff) + (1 - m) * 2 * self.nu * self.alpha[a]
        return diag / self.det, off

    def wall_source(self, k):
        s = torch.zeros_like(self.det)
        for f in range(2 * self.d):
            a = f >> 1
            if (f < 2 and self.periodic_x) or self.ub.get(f) is None:
                continue
            flux = (1.0 if f & 1 else -1.0) * self.det / self.h[a] * self.bound(f, a)
            s = s + (1 - self.mask[f]) * self.bound(f, k) * (2 * self.nu * self.alpha[a] - flux)
        return s / self.det

    def laplace(self, w):
        off = []
        for f in range(2 * self.d):
            c = self.alpha[f >> 1] * w
            off.append(self.mask[f] * 0.5 * (c + self.nb(c, f)))
        return -sum(off), off

    def apply(self, coef, x):
        y = coef[0] * x
        for f in range(2 * self.d):
            y = y + coef[1 + f] * self.nb(x, f)
        return y

    def center(self, x):
        return x - x.mean(dim=(1, 2, 3), keepdim=True)

    def dot(self, a, b):
        return (a * b).sum(dim=(1, 2, 3), keepdim=True)

    def krylov(self, kind, coef, b, tol=1e-13, most=12000):
        """Jacobi-preconditioned CG of the (singular) Laplacians, or BiCGStab with the right-hand
        sides of one instance sharing its matrix; checked every 20 iterations."""
        if kind == "cg":
            b = self.center(b)
            inv = 1.0 / coef[0]
            x = torch.zeros_like(b)
            r, goal = b.clone(), self.dot(b, b) * tol * tol
            z = inv * r
            p, rz = z.clone(), self.dot(r, z)
            for it in range(most):
                q = self.apply(coef, p)
                pq = self.dot(p, q)
                alpha = torch.where(pq != 0, rz / pq, torch.zeros_like(rz))
                x, r = x + alpha * p, r - alpha * q
                z = inv * r
                new = self.dot(r, z)
                p, rz = z + torch.where(rz != 0, new / rz, torch.zeros_like(rz)) * p, new
                if it % 20 == 19 and bool((self.dot(r, r) <= goal).all()):
                    break
            return self.center(x)
        k = b.shape[0] // coef[0].shape[0]
        coef = [c.repeat_interleave(k, 0) if c.shape[0] > 1 else c for c in coef]
        x = torch.zeros_like(b)
        r, goal = b.clone(), self.dot(b, b) * tol * tol
        r0, p, rho = r.clone(), r.clone(), self.dot(b, b)
        zero = torch.zeros_like(rho)

        def safe(n, m):
            return torch.where(m.abs() > 1e-290, n / torch.where(m.abs() > 1e-290, m, torch.ones_like(m)), zero)

        for it in range(600):
            live = self.dot(r, r) > goal
            if it % 5 == 4 and not bool(live.any()):
                break
            v = self.apply(coef, p)
            alpha = torch.where(live, safe(rho, self.dot(r0, v)), zero)
            s = r - alpha * v
            t = self.apply(coef, s)
            omega = torch.where(live, safe(self.dot(t, s), self.dot(t, t)), zero)
            x = x + alpha * p + omega * s
            r = torch.where(live, s - omega * t, r)
            new = self.dot(r0, r)
            beta = torch.where(live, safe(new, rho) * safe(alpha, omega), zero)
            p = torch.where(live, r + beta * (p - omega * v), p)
            rho = torch.where(live, new, rho)
        return x

    def solve(self, kind, diag, off, b):
        if kind == "bicg" and b.dim() == 5:  # [batch, d, z, y, x]
            return _Solve.apply(self, kind, b.reshape((-1,) + b.shape[2:]), diag, *off).view(b.shape)
        return _Solve.apply(self, kind, b, diag, *off)

    def hbya(self, diag, off, u, ustar, src):
        out = []
        for k in range(self.d):
            H = sum(off[f] * self.nb(ustar[k], f) for f in range(2 * self.d))
            out.append((u[k] / self.dt - H + self.wall_source(k) + src[k]) / diag)
        return out

    def divergence(self, v):
        fl = self.fluxes(v)
        return sum(fl[2 * a + 1] - fl[2 * a] for a in range(self.d))

    def correct(self, h, p, diag):
        out = []
        for a in range(self.d):
            lo = torch.where(self.mask[2 * a] > 0, self.nb(p, 2 * a), p)
            hi = torch.where(self.mask[2 * a + 1] > 0, self.nb(p, 2 * a + 1), p)
            fac = torch.where((self.mask[2 * a] > 0) & (self.mask[2 * a + 1] > 0), 0.5, 1.0)
            out.append(h[a] - (hi - lo) * fac / self.h[a] / diag)
        return out

    def cross_eb(self, u, eb):
        u2 = u[2] if self.d > 2 else torch.zeros_like(u[0])
        return [u[1] * eb[2] - u2 * eb[1], u2 * eb[0] - u[0] * eb[2], u[0] * eb[1] - u[1] * eb[0]]

    def epot_rhs(self, x):
        s = torch.zeros_like(x[0])
        for f in range(2 * self.d):
            a = f >> 1
            c = self.det / self.h[a] * x[a]
            wall = c if f in self.open else torch.zeros_like(c)
            s = s + (1.0 if f & 1 else -1.0) * (self.mask[f] * 0.5 * (c + self.nb(c, f)) + (1 - self.mask[f]) * wall)
        return s

    def current(self, phi, x):
        out = []
        for a in range(self.d):
            c = self.det / self.h[a] * x[a]
            j = []
            for f in (2 * a, 2 * a + 1):
                coeff = 0.5 * (self.alpha[a] + self.nb(self.alpha[a], f))
                inner = -coeff * (1.0 if f & 1 else -1.0) * (self.nb(phi, f) - phi) + 0.5 * (c + self.nb(c, f))
                wall = c if f in self.open else torch.zeros_like(c)
                j.append(self.mask[f] * inner + (1 - self.mask[f]) * wall)
            out.append(self.h[a] * 0.5 * (j[0] + j[1]) / self.det)
        if self.d == 2:
            out.append(x[2])
        return out

    def lorentz(self, phi, x, eb, stuart):
        J = self.current(phi, x)
        F = [J[1] * eb[2] - J[2] * eb[1], J[2] * eb[0] - J[0] * eb[2], J[0] * eb[1] - J[1] * eb[0]]
        return [stuart * F[k] for k in range(self.d)]

    def step(self, s, eb, stuart):
        """One PISO step of the state {u, phi, x, scalar}."""
        u = s["u"]
        src = [torch.zeros_like(u[0])] * self.d if stuart is None else self.lorentz(s["phi"], s["x"], eb, stuart)
        diag, off = self.momentum(u)
        out = dict(s)
        if s.get("scalar") is not None:
            out["scalar"] = self.solve("bicg", diag, off, (s["scalar"] / self.dt).unsqueeze(1)).squeeze(1)
        b = torch.stack([u[k] / self.dt + self.wall_source(k) + src[k] for k in range(self.d)], dim=1)
        us = self.solve("bicg", diag, off, b)
        us = [us[:, k] for k in range(self.d)]
        pd, po = self.laplace(1.0 / diag)
        for _ in range(2):
            h = self.hbya(diag, off, u, us, src)
            p = self.solve("cg", pd, po, self.divergence(h))
            us = self.correct(h, p, diag)
        out["u"], out["p"] = us, p
        if stuart is not None:
            x = self.cross_eb(us, eb)
            ed, eo = self.laplace(torch.ones_like(self.det))
            full = torch.ones_like(us[0])
            out["x"], out["phi"] = x, self.solve("cg", ed * full, [o * full for o in eo], self.center(self.epot_rhs(x)))
        return out


_EB = (0.0, 1.0, 0.0)


def _grid(shape, nx, ny, nz, blocks, dt, nu, inflow, device):
    axes = _nodes(shape, nx, ny, nz, blocks)
    ub, open_faces = {}, set()
    if shape == "duct":
        ub = {0: [c.unsqueeze(-1) for c in inflow.unbind(1)]}
        ub[1] = ub[0]
        open_faces = {1}
    elif shape == "cavity":
        ub = {3: [1.0, 0.0]}
    return _Grid(axes, shape in ("channel", "square"), ub, open_faces, dt, nu, device)


def _flat(x, blocks):
    """[batch, z, y, x] to [batch, cells] with the blocks one after another."""
    return torch.cat([c.reshape(x.shape[0], -1) for c in x.chunk(blocks, dim=3)], dim=1)


def _exact_steps(shape, nx, ny, nz, blocks, dts, nus, stuarts, seeds, steps, device, round_to=torch.float64):
    """`steps` steps of instances of one shape: flat u [batch, d * cells], p, phi, scalar."""
    ins = [_inputs(shape, nx, ny, nz, blocks, s, device) for s in seeds]
    u = torch.stack([i[0] for i in ins]).to(round_to).double()
    inflow = torch.stack([i[1] for i in ins]).to(round_to).double() if ins[0][1] is not None else None
    grid = _grid(shape, nx, ny, nz, blocks, dts, nus, inflow, device)
    zero = torch.zeros_like(u[:, 0])
    s = {"u": list(u.unbind(1)), "phi": zero, "x": [zero] * 3}
    if shape == "cavity" and stuarts is None:
        s["scalar"] = torch.stack([i[2] for i in ins]).to(round_to).double()
    N = None if stuarts is None else torch.as_tensor(stuarts, dtype=torch.float64, device=device).view(-1, 1, 1, 1)
    for _ in range(steps):
        s = grid.step(s, _EB, N)
    out = {"u": torch.cat([_flat(c, blocks) for c in s["u"]], dim=1), "p": _flat(s["p"], blocks)}
    if "scalar" in s:
        out["scalar"] = _flat(s["scalar"], blocks)
    if stuarts is not None:
        out["phi"] = _flat(s["phi"], blocks)
    return out


def exact(case, seed):
    device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    k = case["kind"]
    with torch.no_grad():
        if k in ("step", "run"):
            N = None if case["shape"] == "cavity" else [case["ha"] ** 2 / case["re"]]
            # the viscosity is handed over as a float32 tensor, the grid and the fields in the domain's type
            nu = [float(torch.tensor(1.0 / case["re"]))]
            o = _exact_steps(case["shape"], case["nx"], case["ny"], case["nz"], case["blocks"], [case["dt"]], nu, N, [seed],
                             case["steps"] if k == "run" else case["warm"] + 1, device, _dtype(case))
            return {n: v.reshape(-1) for n, v in o.items()}
        if k == "batch":
            mem = _members(case)
            groups = {}
            for e, m in enumerate(mem):
                groups.setdefault(m[:4], []).append(e)
            parts = [None] * len(mem)
            for (shape, nx, ny, nz), es in groups.items():
                o = _exact_steps(shape, nx, ny, nz, 1, [mem[e][6] for e in es], [float(torch.tensor(1.0 / mem[e][4])) for e in es],
                                 [mem[e][5] for e in es], [seed * 1000 + e for e in es], case["warm"] + 1, device)
                for i, e in enumerate(es):
                    parts[e] = {n: v[i].reshape(-1) for n, v in o.items()}
            return {n: torch.cat([p[n] for p in parts]) for n in ("u", "p", "phi")}
        if k == "assembly":
            return _exact_assembly(case, seed, device)
    return _exact_gradient(case, seed, device)


def _exact_gradient(case, seed, device):
    shape = ("duct", case["nx"], case["ny"], case["nz"], case["blocks"])
    u, inflow, _ = _inputs(*shape, seed, device)
    prof = inflow.unsqueeze(0).requires_grad_(True)
    N = torch.tensor([case["ha"] ** 2 / case["re"]], dtype=torch.float64, device=device, requires_grad=True)
    grid = _grid(*shape, [case["dt"]], [float(torch.tensor(1.0 / case["re"]))], prof, device)
    zero = torch.zeros_like(u[:1])
    s = {"u": [c.unsqueeze(0) for c in u.unbind(0)], "phi": zero, "x": [zero] * 3}
    for _ in range(case["steps"]):
        s = grid.step(s, _EB, N.view(-1, 1, 1, 1))
    uf = torch.cat([_flat(c, case["blocks"]) for c in s["u"]], dim=1).reshape(-1)
    (uf * _loss_weight(case, seed, device)).sum().backward()
    return {"u": uf.detach(), "profile_grad": prof.grad.reshape(1, 3, case["nz"], case["ny"], 1), "stuart_grad": N.grad.cpu()}


def _exact_assembly(case, seed, device):
    dt = _dtype(case)
    shape = "duct" if case["dims"] == 3 else "square"
    size = (shape, case["nx"], case["ny"], case["nz"], 1)
    u, inflow, _ = _inputs(*size, seed, device)
    inflow = None if inflow is None else inflow.to(dt).double().unsqueeze(0)
    grid = _grid(*size, [1e-3], [float(torch.tensor(1e-3))], inflow, device)
    if dt == torch.float32:  # the product sees the vertices in float32
        axes = [np.asarray(a, dtype=np.float32).astype(np.float64) for a in _nodes(*size)]
        grid = _Grid(axes, shape == "square", grid.ub, grid.open, [1e-3], [float(torch.tensor(1e-3))], device)
    f = {n: v.to(dt).double().unsqueeze(0) for n, v in _assembly_fields(case, seed, device).items()}
    uu = list(u.to(dt).double().unsqueeze(0).unbind(1))
    src = list(f["src"].unbind(1))
    diag, off = grid.momentum(uu)
    d = case["dims"]
    out = {"C": torch.stack([c.expand_as(uu[0]).reshape(-1) for c in [diag] + off]), "A": diag.reshape(-1)}
    out["rhs"] = torch.cat([(uu[k] / grid.dt + grid.wall_source(k) + src[k]).reshape(-1) for k in range(d)])
    pd, po = grid.laplace(1.0 / diag)
    out["P"] = torch.stack([c.reshape(-1) for c in [pd] + po])
    del pd, po
    h = grid.hbya(diag, off, uu, uu, src)
    out["hbya"] = torch.cat([c.reshape(-1) for c in h])
    out["div"] = grid.divergence(h).reshape(-1)
    out["u"] = torch.cat([c.reshape(-1) for c in grid.correct(h, f["p"], diag)])
    x = list(f["uxb"].unbind(1))
    out["epot_rhs"] = grid.epot_rhs(x).reshape(-1)
    out["J"] = torch.cat([c.reshape(-1) for c in grid.current(f["phi"], x)])
    return out
