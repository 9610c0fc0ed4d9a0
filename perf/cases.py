"""The framework's working range as timed cases: time steps of single and batched simulations, of a multi-block
street and of a 3D channel, gradients of rollouts, the operators a user's own loop calls, scalar transport and
multi-block padding.

``listed()`` names the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare`` builds what a program has
in hand (domain, fields, stepper, captured graph), ``run`` is one pass through the public entry points, ``work`` the
bytes and operations of a pass, ``tolerance`` how far a correct result may be from another one, and ``exact`` the
result in 64 bits from plain torch (class ``Flow64``), for the inputs as they are given in the case's data type.

A pass of a stepping case loads the prepared fields and takes ``steps`` time steps from them, so every pass is the
same work: a window of a simulation, as a driver, a data generator or a training loop takes it.
"""
import math

import numpy as np
import torch

from pict_b200 import PISOtorch as P
from pict_b200.adjoint import PISOAdjoint, rollout
from pict_b200.batch import BatchDomain
from pict_b200.cylinder_street import TIME_STEP, build_street, street_spec
from pict_b200.engine import PISOStepper
from pict_b200.multiblock_cnn import MultiblockConv
from pict_b200.PISOtorch_simulation import Simulation

WARM = 4          # steps a batch takes before its fields are kept as the pass' start (past the impulsive lid)
SKEW_FLAGS = 25   # non-orthogonal terms as the Simulation driver takes them: centre and direct matrix, diagonal RHS


def listed():
    return [
        # the reference's minimal sample: one 64^2 lid-driven cavity in FP32; latency and launches count
        dict(name="cavity_64", kind="cavities", num=1, lo=64, hi=64, size_seed=0, mixed=False, steps=8),
        # the drop-in Simulation class on a small 3D cavity in FP64 with its default settings
        dict(name="simulation_3d_f64", kind="simulation", n=32, steps=2),
        # a few simulations of uneven size in mixed precision
        dict(name="cavities_16", kind="cavities", num=16, lo=32, hi=256, size_seed=16, mixed=True, steps=4),
        # the benchmark's batch: 256 simulations, 32 to 256 cells a side
        dict(name="cavities_256", kind="cavities", num=256, lo=32, hi=256, size_seed=6, mixed=True, steps=4),
        # multi-block flow past a cylinder with the advective outflow, FP32 with refined pressure, solves from zero
        dict(name="street", kind="street", n=64, steps=2),
        # wall-stretched 3D channel, mixed precision refined to 1e-10
        dict(name="channel_192", kind="channel", nx=192, ny=96, nz=96, steps=3),
        # forward and backward through the checkpointed rollout of a batch (viscosity and initial velocity)
        dict(name="gradient_64", kind="gradient", num=64, lo=32, hi=256, size_seed=64, steps=4, window=2),
        # learning a per-cell forcing on the 128^2 periodic box, FP64
        dict(name="forcing_128_f64", kind="forcing", n=128, steps=4, window=4),
        # the operators of a user's own loop on a ragged curvilinear 2D grid, FP32
        dict(name="operators_2d", kind="operators", nx=1021, ny=773),
        # the operators with the non-orthogonal terms on a wavy 3D grid, FP64
        dict(name="skewed_3d_f64", kind="skewed", nx=96, ny=65, nz=80),
        # two passive scalars and the sub-grid viscosity in a 3D channel, FP32
        dict(name="scalars_3d", kind="scalars", nx=120, ny=64, nz=72, steps=1),
        # multi-block convolution padding, forward and backward, on a 2x2 grid of blocks
        dict(name="padding", kind="padding", m=512, batch=4, channels=16, kernel=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cavities", "cavities", "simulation", "street", "channel", "gradient", "forcing", "operators",
                       "skewed", "scalars", "padding"])
    if kind == "cavities":
        num = _log(rng, 1, 224)
        if num < 4 and rng.random() < 0.5:
            n = _log(rng, 24, 256)
            return dict(kind=kind, num=num, lo=n, hi=n, size_seed=rng.randrange(1000), mixed=False, steps=4)
        return dict(kind=kind, num=num, lo=rng.randrange(24, 48), hi=rng.randrange(96, 257),
                    size_seed=rng.randrange(1000), mixed=True, steps=4)
    if kind == "simulation":
        return dict(kind=kind, n=_log(rng, 10, 48), steps=2)
    if kind == "street":
        return dict(kind=kind, n=2 * rng.randrange(8, 33), steps=2)
    if kind == "channel":
        s = math.exp(rng.uniform(math.log(0.25), 0.0))
        return dict(kind=kind, nx=max(16, int(192 * s)), ny=max(12, int(96 * s * rng.uniform(0.8, 1.0))),
                    nz=max(12, int(96 * s * rng.uniform(0.8, 1.0))), steps=3)
    if kind == "gradient":
        return dict(kind=kind, num=_log(rng, 2, 64), lo=rng.randrange(24, 48), hi=rng.randrange(96, 225),
                    size_seed=rng.randrange(1000), steps=4, window=rng.choice([2, 4]))
    if kind == "forcing":
        return dict(kind=kind, n=_log(rng, 32, 144), steps=4, window=rng.choice([2, 4]))
    if kind == "operators":
        return dict(kind=kind, nx=_log(rng, 40, 1400), ny=_log(rng, 40, 1400))
    if kind == "skewed":
        return dict(kind=kind, nx=_log(rng, 12, 110), ny=_log(rng, 12, 90), nz=_log(rng, 12, 90))
    if kind == "scalars":
        return dict(kind=kind, nx=_log(rng, 16, 130), ny=_log(rng, 12, 72), nz=_log(rng, 12, 72), steps=1)
    return dict(kind="padding", m=_log(rng, 24, 512), batch=rng.randrange(1, 5), channels=rng.choice([2, 3, 8, 16]),
                kernel=rng.choice([3, 5]))


# ---------------------------------------------------------------------------------------------- inputs

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _dtype(c):
    return torch.float64 if c["kind"] in ("simulation", "forcing", "skewed") else torch.float32


def _t(a, dtype):
    return torch.as_tensor(a, dtype=torch.float64).to(_dev()).to(dtype).contiguous()


def _grid(*axes):
    """Vertex coordinates [1, D, (z), y, x] of a tensor-product grid from the x, y(, z) vertex positions."""
    g = np.meshgrid(*axes[::-1], indexing="ij")
    return np.stack(g[::-1])[None]


def _stretched(n, beta=2.0):
    s = np.linspace(-1.0, 1.0, n + 1)
    return np.tanh(beta * s) / np.tanh(beta)


def _swirl(coords, rng, periodic=False, amplitude=0.5, modes=6):
    """Seeded smooth divergence-free field [1, 2, y, x] at the cell centres of a unit box: a stream function of a
    few modes that vanishes on the walls (or is periodic), as the fields a cavity or a periodic box holds."""
    xy = torch.as_tensor(coords[0], device=_dev())
    c = 0.25 * (xy[:, 1:, 1:] + xy[:, 1:, :-1] + xy[:, :-1, 1:] + xy[:, :-1, :-1])
    u = torch.zeros_like(c)
    for _ in range(modes):
        a, ph = rng.standard_normal(), rng.uniform(0, 2 * np.pi)
        kx, ky = rng.integers(1, 5), rng.integers(1, 5)
        a = a / (kx * kx + ky * ky)
        if periodic:
            arg = 2 * np.pi * (kx * c[0] + ky * c[1]) + ph
            u[0] -= a * ky * torch.sin(arg)
            u[1] += a * kx * torch.sin(arg)
        else:
            x, y = np.pi * kx * c[0], np.pi * ky * c[1]
            u[0] += a * ky * torch.sin(x) * torch.cos(y)
            u[1] -= a * kx * torch.cos(x) * torch.sin(y)
    return (u * (amplitude / u.abs().max()))[None]


def _noise(shape, rng, scale=1.0):
    return rng.standard_normal(shape) * scale


def _batch_params(c, seed):
    """Sides (fixed by the case), viscosities and initial velocities (from the seed) of a batch of cavities."""
    sides = np.rint(np.exp(np.random.default_rng(c["size_seed"]).uniform(math.log(c["lo"]), math.log(c["hi"]),
                                                                         c["num"]))).astype(int)
    rng = np.random.default_rng(seed)
    re = np.exp(rng.uniform(math.log(100), math.log(5000), c["num"]))
    out = []
    for s, r in zip(sides, re):
        co = _grid(np.linspace(0, 1, s + 1), np.linspace(0, 1, s + 1))
        out.append(dict(coords=_t(co, torch.float32), nu=float(np.float32(1.0 / r)), dt=float(np.float32(0.5 / s)),
                        u=_swirl(co, rng).float()))
    return out


def _inputs(c, seed):
    """Inputs of a case in its data type, from the seed alone (the same for the framework and for `exact`)."""
    k, rng, dt = c["kind"], np.random.default_rng(seed), _dtype(c)
    if k == "simulation":
        x = np.linspace(0, 1, c["n"] + 1)
        u = _noise((1, 3, c["n"], c["n"], c["n"]), rng, 0.02)
        return dict(coords=_t(_grid(x, x, x), dt), u=_t(u, dt))
    if k == "channel":
        x, y, z = np.linspace(0, 4 * np.pi, c["nx"] + 1), _stretched(c["ny"]), np.linspace(0, 4 * np.pi / 3, c["nz"] + 1)
        yc, xc = torch.as_tensor(0.5 * (y[1:] + y[:-1])), torch.as_tensor(0.5 * (x[1:] + x[:-1]))
        zc = torch.as_tensor(0.5 * (z[1:] + z[:-1]))
        Z, Y, X = [g.to(_dev()) for g in torch.meshgrid(zc, yc, xc, indexing="ij")]
        u = torch.zeros((1, 3) + tuple(X.shape), dtype=torch.float64, device=_dev())
        u[0, 0] = 20.0 * (1 - Y ** 2)
        for _ in range(6):  # streamwise vortices and oblique waves, zero at the walls
            kx, kz, ph = 0.5 * rng.integers(1, 4), 1.5 * rng.integers(1, 4), rng.uniform(0, 2 * np.pi)
            w, a = (1 - Y ** 2) ** 2, rng.standard_normal() * 0.5
            arg = kx * X + kz * Z + ph
            u[0, 0] += a * kz * w * torch.cos(arg)
            u[0, 2] -= a * kx * w * torch.cos(arg)
        return dict(coords=_t(_grid(x, y, z), dt), u=u.to(dt).contiguous())
    if k == "forcing":
        x = np.linspace(0, 1, c["n"] + 1)
        co = _grid(x, x)
        return dict(coords=_t(co, dt), u=_swirl(co, rng, True).to(dt).contiguous(),
                    f=(0.2 * _swirl(co, rng, True)).to(dt).contiguous(), target=_swirl(co, rng, True).to(dt))
    if k == "operators":
        co = _grid(np.linspace(0, 2, c["nx"] + 1), 0.75 * (1 + _stretched(c["ny"], 1.5)))
        bump = 0.05 * np.sin(np.pi * co[0, 0] / 2) * np.sin(np.pi * co[0, 1] / 1.5)
        co[0, 0] += bump
        co[0, 1] -= 0.5 * bump
        shape = (c["ny"], c["nx"])
        return dict(coords=_t(co, dt), u=_t(_noise((1, 2) + shape, rng, 0.3), dt), p=_t(_noise((1, 1) + shape, rng), dt),
                    us=_t(_noise((1, 2) + shape, rng, 0.3), dt))
    if k == "skewed":
        co = _grid(*[np.linspace(0, 1, c[a] + 1) for a in ("nx", "ny", "nz")])
        X, Y, Z = co[0].copy()
        co[0, 0] += 0.04 * np.sin(2 * np.pi * Y) + 0.2 * Y
        co[0, 1] += 0.03 * np.sin(2 * np.pi * Z) * np.cos(2 * np.pi * X)
        co[0, 2] += 0.04 * np.cos(2 * np.pi * X)
        shape = (c["nz"], c["ny"], c["nx"])
        return dict(coords=_t(co, dt), u=_t(_noise((1, 3) + shape, rng, 0.3), dt), p=_t(_noise((1, 1) + shape, rng), dt))
    if k == "scalars":
        x, y, z = np.linspace(0, 4 * np.pi, c["nx"] + 1), _stretched(c["ny"], 1.5), np.linspace(0, 4 * np.pi / 3, c["nz"] + 1)
        shape = (c["nz"], c["ny"], c["nx"])
        u = _noise((1, 3) + shape, rng, 0.1)
        u[0, 0] += (1 - (0.5 * (y[1:] + y[:-1])) ** 2)[None, :, None]
        return dict(coords=_t(_grid(x, y, z), dt), u=_t(u, dt), s=_t(rng.random((1, 2) + shape), dt))
    g = torch.Generator(device=_dev()).manual_seed(int(seed))
    shape = (c["batch"], c["channels"])
    p2 = c["kernel"] - 1
    sizes = _padding_sizes(c["m"])
    return dict(x=[torch.randn(shape + s, generator=g, device=_dev()) for s in sizes],
                g=[torch.randn(shape + (s[0] + p2, s[1] + p2), generator=g, device=_dev()) for s in sizes])


def _padding_sizes(m):
    """(y, x) sizes of the 2x2 grid of blocks: columns m and m - 5 wide, rows m and m + 3 high."""
    return [(m, m), (m, m - 5), (m + 3, m), (m + 3, m - 5)]


# ---------------------------------------------------------------------------------------------- the framework's side

def _domain(dims, nu, dtype, coords, u=None, channels=0, scalar=None, scalar_viscosity=None):
    dom = P.Domain(dims, torch.tensor([nu], dtype=dtype), name="case", dtype=dtype, device=_dev(),
                   passiveScalarChannels=channels, scalarViscosity=scalar_viscosity)
    kw = {} if scalar is None else dict(passiveScalar=scalar.clone())
    blk = dom.CreateBlock(velocity=None if u is None else u.clone(), vertexCoordinates=coords, name="block", **kw)
    return dom, blk


def _lid(dims, dtype):
    return _t([[1.0] + [0.0] * (dims - 1)], dtype)


def _batch(c, seed):
    doms, dts = [], []
    for b in _batch_params(c, seed):
        dom, blk = _domain(2, b["nu"], torch.float32, b["coords"], b["u"])
        blk.CloseAllBoundaries()
        blk.CloseBoundary("-y", _lid(2, torch.float32))
        dom.PrepareSolve()
        doms.append(dom)
        dts.append(b["dt"])
    batch = BatchDomain(doms, time_steps=dts)
    batch.pack_state()
    if c.get("mixed", True):
        kw = dict(advection_tol=5e-7, pressure_refine=1, refine_tol=5e-10, warm_start_pressure="increment",
                  refine_solver="auto", mg_iterations=16, pressure_first_solve=False, warm_start_advection="increment")
    else:
        kw = dict(advection_tol=1e-6)
    return batch, PISOStepper(batch, time_step=dts[0], corrector_steps=2, pressure_tol=1e-6, **kw)


def _channel(c, seed):
    i = _inputs(c, seed)
    dom, blk = _domain(3, 1.0 / 180.0, torch.float32, i["coords"], i["u"])
    blk.MakePeriodic("x")
    blk.MakePeriodic("z")
    blk.CloseBoundary("-y")
    blk.CloseBoundary("+y")
    blk.setVelocitySource(_t([[1.0, 0.0, 0.0]], torch.float32))
    dom.PrepareSolve()
    return dom, PISOStepper(dom, time_step=_channel_dt(c), corrector_steps=2, advection_tol=1e-6, pressure_tol=1e-6,
                            pressure_refine=1, refine_tol=1e-10, warm_start_pressure="increment", refine_solver="auto",
                            pressure_first_solve=False, warm_start_advection="increment")


def _channel_dt(c):
    return 0.5 * (4 * math.pi / c["nx"]) / 20.0


def _street_spec(c, seed):
    """The street of n x n cells per quadrant with a seeded inflow; the outflow starts with the inflow's flux."""
    spec = street_spec(n_ang=c["n"], n_rad=c["n"], dx=8.0 / c["n"], inflow_seed=int(seed))
    op = {(o[1], o[2]): o for o in spec["ops"] if o[0] == "close"}
    dy = np.diff(spec["blocks"][4]["coords"][0, 1, :, 0])
    op[spec["outflow"][0][0], "+x"][3][0, 0] = (op[4, "-x"][3][0, 0, :, 0] * dy).sum() / dy.sum()
    return spec


def _padding_layer(c):
    sizes = _padding_sizes(c["m"])
    dom = P.Domain(2, torch.tensor([1e-3]), name="grid", dtype=torch.float32, device=_dev(), passiveScalarChannels=0)
    b = [dom.CreateBlockWithSize(P.Int4(s[1], s[0], 1, 2), name="b%d" % i) for i, s in enumerate(sizes)]
    for x in b:
        x.CloseAllBoundaries()
    b[0].ConnectBlock("+x", b[1], "-x", "-y")
    b[0].ConnectBlock("+y", b[2], "-y", "-x")
    b[1].ConnectBlock("+y", b[3], "-y", "-x")
    b[2].ConnectBlock("+x", b[3], "-x", "-y")
    return MultiblockConv(dom, "ZERO", c["channels"], c["channels"], c["kernel"], device=_dev(), dtype=torch.float32)


def prepare(case, seed):
    c, k = case, case["kind"]
    if k == "cavities":
        batch, st = _batch(c, seed)
        for _ in range(WARM):
            st.step()
        st.check()
        st.capture(steps=1)
        return dict(c=c, dom=batch, st=st, u0=batch.velocity_arena.clone())
    if k == "channel":
        dom, st = _channel(c, seed)
        for _ in range(2):
            st.step()
        st.check()
        st.capture(steps=1)
        return dict(c=c, dom=dom, st=st, u0=dom.getBlock(0).velocity.clone())
    if k == "street":
        dom, info = build_street(_street_spec(c, seed), dtype=torch.float32)
        st = PISOStepper(dom, time_step=TIME_STEP, advection_tol=1e-6, pressure_tol=1e-6, pressure_refine=1,
                         refine_tol=1e-8, outflow=info["outflow"], outflow_velocity=info["char_vel"])
        for _ in range(2):
            st.step()
        st.check()
        st.capture(steps=1)
        out = [dom.getBlock(b).getBoundary(f) for b, f in info["outflow"]]
        return dict(c=c, dom=dom, st=st, u0=[b.velocity.clone() for b in dom.getBlocks()],
                    out=out, out0=[o.velocity.clone() for o in out])
    if k == "gradient":
        batch, st = _batch(c, seed)
        adj = PISOAdjoint(st, relative_tolerance=True, adjoint_pressure_tol=1e-6)
        u0 = adj.velocity().clone()
        for _ in range(WARM):
            st.step()
        st.check()
        st.capture(steps=1)
        adj.use_graph = True
        n = torch.tensor([batch.domains[i].getTotalSize() for i in batch.order], device=_dev())
        w = torch.repeat_interleave(1.0 / (n.numel() * n.float()), n).repeat(2)
        nu = torch.tensor([float(batch.domains[i].viscosity) for i in batch.order], device=_dev())
        return dict(c=c, adj=adj, st=st, dom=batch, u0=u0, nu=nu, w=w)
    if k == "forcing":
        i = _inputs(c, seed)
        dom, blk = _domain(2, 1e-3, torch.float64, i["coords"], i["u"])
        blk.setVelocitySource(i["f"].clone())
        dom.PrepareSolve()
        st = PISOStepper(dom, time_step=0.5 / c["n"])
        adj = PISOAdjoint(st, relative_tolerance=True)
        st.capture(steps=1)
        adj.use_graph = True
        return dict(c=c, adj=adj, st=st, dom=dom, u0=i["u"].reshape(-1), f=i["f"].reshape(-1), target=i["target"].reshape(-1))
    i = _inputs(c, seed)
    if k == "simulation":
        dom, blk = _domain(3, 1e-2, torch.float64, i["coords"], i["u"])
        blk.CloseAllBoundaries()
        blk.CloseBoundary("+y", _lid(3, torch.float64))
        dom.PrepareSolve()
        sim = Simulation(domain=dom, time_step=0.2 / c["n"], corrector_steps=2, non_orthogonal=False)
        return dict(c=c, dom=dom, sim=sim, u0=i["u"])
    if k == "operators":
        dom, blk = _domain(2, 1e-3, torch.float32, i["coords"], i["u"])
        blk.CloseAllBoundaries()
        blk.CloseBoundary("-y", _lid(2, torch.float32))
        blk.setPressure(i["p"])
        dom.PrepareSolve()
        return dict(c=c, dom=dom, us=i["us"].reshape(-1), dt=torch.tensor([0.5 / c["nx"]]))
    if k == "skewed":
        dom, blk = _domain(3, 1e-3, torch.float64, i["coords"], i["u"])
        blk.setPressure(i["p"])
        dom.PrepareSolve()
        return dict(c=c, dom=dom, dt=torch.tensor([0.5 / c["nx"]], dtype=torch.float64))
    if k == "scalars":
        dom, blk = _domain(3, 1e-3, torch.float32, i["coords"], i["u"], 2, i["s"], _t([2e-3], torch.float32))
        blk.MakePeriodic("x")
        blk.MakePeriodic("z")
        blk.CloseBoundary("-y", None, _t([[1.0, 0.5]], torch.float32))
        blk.CloseBoundary("+y", None, _t([[0.0, 0.0]], torch.float32))
        dom.PrepareSolve()
        sim = Simulation(domain=dom, time_step=_scalar_dt(c), corrector_steps=2, advection_tol=1e-6, non_orthogonal=False,
                         advect_passive_scalar=True)
        return dict(c=c, dom=dom, sim=sim, s0=i["s"], coef=torch.tensor([0.17 ** 2]))
    return dict(c=c, layer=_padding_layer(c), x=i["x"], g=i["g"])


def _scalar_dt(c):
    return 0.5 * (4 * math.pi / c["nx"])


def run(state):
    s = state
    c, k = s["c"], s["c"]["kind"]
    if k == "cavities":
        s["dom"].velocity_arena.copy_(s["u0"])
        for _ in range(c["steps"]):
            s["st"].replay()
        return s["dom"].velocity_arena, s["dom"].pressure_arena
    if k == "channel":
        b = s["dom"].getBlock(0)
        b.velocity.copy_(s["u0"])
        for _ in range(c["steps"]):
            s["st"].replay()
        return b.velocity, b.pressure
    if k == "street":
        for b, u in zip(s["dom"].getBlocks(), s["u0"]):
            b.velocity.copy_(u)
        for o, u in zip(s["out"], s["out0"]):
            o.velocity.copy_(u)
        for _ in range(c["steps"]):
            s["st"].replay()
        blocks = s["dom"].getBlocks()
        return dict(u=torch.cat([b.velocity.reshape(2, -1) for b in blocks], dim=1),
                    p=torch.cat([b.pressure.reshape(-1) for b in blocks]), out=s["out"][0].velocity)
    if k == "gradient":
        u0, nu = s["u0"].clone().requires_grad_(True), s["nu"].clone().requires_grad_(True)
        (u,) = rollout(s["adj"], u0, c["steps"], [c["steps"]], checkpoint_every=c["window"], nu=nu)
        (0.5 * (s["w"] * u * u).sum()).backward()
        return dict(u=u.detach(), grad_u=u0.grad, grad_nu=nu.grad)
    if k == "forcing":
        f = s["f"].clone().requires_grad_(True)
        rec = sorted({c["steps"] // 2, c["steps"]})
        outs = rollout(s["adj"], s["u0"], c["steps"], rec, checkpoint_every=c["window"], src=f)
        sum(((o - s["target"]) ** 2).mean() for o in outs).backward()
        return dict(u=[o.detach() for o in outs], grad=f.grad)
    dom = s.get("dom")
    if k == "simulation":
        b = dom.getBlock(0)
        b.velocity.copy_(s["u0"])
        s["sim"].run(iterations=c["steps"])
        return b.velocity, b.pressure
    if k == "operators":
        P.SetupAdvectionMatrix(dom, s["dt"], 0)
        P.SetupAdvectionVelocity(dom, s["dt"], 0)
        dom.velocityResult.copy_(s["us"])
        P.SetupPressureCorrection(dom, s["dt"])
        P.CorrectVelocity(dom, s["dt"], 1)
        return dict(A=dom.A, C=dom.C.coef, rhs=dom.velocityRHS, P=dom.P.coef, h=dom.pressureRHS, div=dom.pressureRHSdiv,
                    u=dom.velocityResult, udiv=P.ComputeVelocityDivergence(dom))
    if k == "skewed":
        P.SetupAdvectionMatrix(dom, s["dt"], SKEW_FLAGS)
        P.CopyVelocityResultFromBlocks(dom)
        P.SetupAdvectionVelocity(dom, s["dt"], SKEW_FLAGS)
        P.CopyPressureResultFromBlocks(dom)
        P.SetupPressureMatrix(dom, s["dt"], SKEW_FLAGS)
        P.SetupPressureRHS(dom, s["dt"], SKEW_FLAGS)
        return dict(A=dom.A, C=dom.C.coef, rhs=dom.velocityRHS, P=dom.P.coef, h=dom.pressureRHS, div=dom.pressureRHSdiv)
    if k == "scalars":
        b = dom.getBlock(0)
        b.passiveScalar.copy_(s["s0"])
        s["sim"].run(iterations=c["steps"], static=True)
        return dict(s=b.passiveScalar, nu=P.SGSviscosityIncompressibleSmagorinsky(dom, s["coef"]))
    x = [t.detach().requires_grad_(True) for t in s["x"]]
    y = s["layer"].pad(x)
    torch.autograd.backward(y, s["g"])
    return dict(y=[t.detach() for t in y], grad=[t.grad for t in x])


# ---------------------------------------------------------------------------------------------- work and tolerance

def _cells(c):
    k = c["kind"]
    if k in ("cavities", "gradient"):
        s = np.rint(np.exp(np.random.default_rng(c["size_seed"]).uniform(math.log(c["lo"]), math.log(c["hi"]), c["num"])))
        return int((s.astype(int) ** 2).sum())
    if k == "simulation":
        return c["n"] ** 3
    if k == "street":
        n = c["n"]
        return 4 * n * n + n * (n // 2) + 3 * n * int(round(0.75 * n))
    if k == "forcing":
        return c["n"] ** 2
    if k == "operators":
        return c["nx"] * c["ny"]
    if k == "padding":
        return sum(a * b for a, b in _padding_sizes(c["m"]))
    return c["nx"] * c["ny"] * c["nz"]


def work(case):
    """A time step reads the velocity and the metrics and writes velocity and pressure; what a solve moves between
    its first read and its last write is not counted.  A gradient reads and writes the same fields once more."""
    c, k, n = case, case["kind"], _cells(case)
    e = 8 if _dtype(c) == torch.float64 else 4
    D = 3 if k in ("simulation", "channel", "skewed", "scalars") else 2
    t, K = 2 * D * D + 1, 2 * D + 1
    if k == "padding":
        pad = sum((a + c["kernel"] - 1) * (b + c["kernel"] - 1) for a, b in _padding_sizes(c["m"]))
        return dict(bytes=e * 2 * c["batch"] * c["channels"] * (n + pad), flops=c["batch"] * c["channels"] * pad)
    if k == "operators":  # u, u*, p and metrics in; A, C, rhs, P, h, div, u and its divergence out
        return dict(bytes=e * n * (2 * D + 1 + t + 1 + K + D + K + D + 1 + D + 1), flops=n * (40 * D + 60))
    if k == "skewed":
        return dict(bytes=e * n * (D + 1 + t + 1 + K + D + K + D + 1), flops=n * 600)
    if k == "scalars":
        return dict(bytes=e * n * (c["steps"] * (D + 2 + t + 2) + D + t + 1), flops=n * (300 * c["steps"] + 80))
    step = e * n * (2 * D + 1 + t)
    passes = c["steps"] * (2 if k in ("gradient", "forcing") else 1)
    return dict(bytes=step * passes, flops=n * 60 * (D + 1) * passes)


def tolerance(case):
    if case["kind"] == "cavities" and not case["mixed"]:
        return {"rel": 1e-2, "max": 0.2}
    return TOLERANCE[case["kind"]]


# Steps: the solves stop at a residual, so two correct solves may be as far apart as either is from the exact
# solution (pressure: 1e-3 .. 2e-2 for FP32 solves to 1e-6, 1e-4 refined batches, 7e-4 channel, 1e-3 the FP64 default),
# and another summation order or recurrence was 1e-5 .. 4e-4 away.  Operators: rounding of the data type.
TOLERANCE = {
    "cavities": {"rel": 5e-4, "max": 2e-2},
    "simulation": {"rel": 5e-3, "max": 0.1},
    "street": {"rel": 1e-2, "max": 0.2},
    "channel": {"rel": 3e-3, "max": 5e-2},
    "gradient": {"rel": 1e-5, "max": 1e-3},
    "forcing": {"rel": 5e-5, "max": 5e-3},
    "operators": {"rel": 1e-5, "max": 1e-3},
    "skewed": {"rel": 1e-13, "max": 1e-11},
    "scalars": {"rel": 3e-6, "max": 1e-4},
    "padding": {"rel": 1e-6, "max": 1e-5},
}


# ---------------------------------------------------------------------------------------------- 64 bits

class Flow64:
    """The PISO discretisation in FP64 torch over a flat list of cells: blocks given by vertex coordinates
    [D, (z), y, x] and faces (None: periodic, an array: prescribed velocity [D] or [D, face cells], a tuple
    (block, face, inverted): connected, 2D).  Linear systems are solved to round-off with Jacobi-preconditioned
    CG and BiCGStab over all cells at once."""

    def __init__(self, blocks, nu, dt, source=None):
        dev = _dev()
        D = self.D = blocks[0]["coords"].shape[0]
        F = 2 * D
        n = [int(np.prod([s - 1 for s in b["coords"].shape[1:]])) for b in blocks]
        off = np.concatenate([[0], np.cumsum(n)])
        N = self.N = int(off[-1])
        idx = [torch.arange(int(off[i]), int(off[i + 1]), device=dev).reshape([s - 1 for s in b["coords"].shape[1:]])
               for i, b in enumerate(blocks)]
        self.sim = torch.repeat_interleave(torch.arange(len(n), device=dev), torch.tensor(n, device=dev))
        if not all(isinstance(f, (type(None), torch.Tensor)) for b in blocks for f in b["faces"]):
            self.sim = torch.zeros_like(self.sim)  # connected blocks are one system
        self.ns = int(self.sim.max()) + 1
        self.count = torch.zeros(self.ns, dtype=torch.float64, device=dev).index_add_(
            0, self.sim, torch.ones(N, dtype=torch.float64, device=dev))
        z = lambda *s: torch.zeros(s, dtype=torch.float64, device=dev)
        self.M = z(N, D, D)
        self.nb = torch.empty((F, N), dtype=torch.long, device=dev)
        self.fixed = torch.zeros((F, N), dtype=torch.bool, device=dev)
        self.bvel, self.bflux, self.balpha = z(F, D, N), z(F, N), z(F, N)
        comp = torch.arange(F, device=dev).div(2, rounding_mode="floor")[:, None].repeat(1, N)
        flip = torch.ones((F, N), dtype=torch.float64, device=dev)
        self.bfaces = {}
        for i, b in enumerate(blocks):
            v = b["coords"].double().to(dev)
            cols = torch.stack([self._edges(v, a, None) for a in range(D)])        # [k, D, cells]
            self.M[off[i]:off[i + 1]] = cols.reshape(D, D, -1).permute(2, 1, 0)
            for f in range(F):
                a, up = f >> 1, f & 1
                ax = D - 1 - a
                last = idx[i].shape[ax] - 1
                own = idx[i].narrow(ax, last if up else 0, 1)
                face = b["faces"][f]
                if face is None:
                    edge = idx[i].narrow(ax, 0 if up else last, 1)
                elif isinstance(face, tuple):
                    ob, of, inv = face
                    oax = D - 1 - (of >> 1)
                    edge = idx[ob].select(oax, idx[ob].shape[oax] - 1 if of & 1 else 0)
                    edge = (edge.flip(0) if inv else edge).reshape(own.shape)
                    comp[f][own.reshape(-1)] = of >> 1
                    flip[f][own.reshape(-1)] = -1.0 if (of & 1) == up else 1.0
                else:
                    edge = own
                    o = own.reshape(-1)
                    self.fixed[f][o] = True
                    t = torch.stack([cols[k].narrow(ax + 1, last if up else 0, 1) if k == a else self._edges(v, k, (a, up))
                                     for k in range(D)]).reshape(D, D, -1).permute(2, 1, 0)
                    self.bfaces[(i, f)] = (o, t)
                    self.set_face(i, f, face.double().to(dev))
                rest = idx[i].narrow(ax, 1 if up else 0, last)
                self.nb[f][idx[i].reshape(-1)] = torch.cat([rest, edge] if up else [edge, rest], dim=ax).reshape(-1)
        self.Minv, self.det = torch.linalg.inv(self.M), torch.linalg.det(self.M)
        self.Wc = [self.det[:, None] * self.Minv[:, a] for a in range(D)]
        self.Wn = [(flip[f] * self.det[self.nb[f]])[:, None] * self.Minv[self.nb[f], comp[f]] for f in range(F)]
        self.alpha = [self.det * (self.Minv[:, a] ** 2).sum(1) for a in range(D)]
        self.alphaN = [(self.Wn[f] ** 2).sum(1) / self.det[self.nb[f]] for f in range(F)]
        self.nu, self.dt = nu, dt
        self.src = z(D, 1) if source is None else source

    def _edges(self, v, k, face):
        """Mean edge vector along axis k of every cell (face None) or of every cell of a block face (axis, upper)."""
        D = self.D
        if face is not None:
            ax = D - face[0]
            v = v.narrow(ax, v.shape[ax] - 1 if face[1] else 0, 1)
        d = v.diff(dim=D - k)
        for a in range(D):
            if a != k and not (face is not None and a == face[0]):
                ax = D - a
                m = d.shape[ax] - 1
                d = 0.5 * (d.narrow(ax, 0, m) + d.narrow(ax, 1, m))
        return d

    def set_face(self, i, f, vel):
        o, M = self.bfaces[(i, f)]
        a, inv, det = f >> 1, torch.linalg.inv(M), torch.linalg.det(M)
        v = (vel.reshape(self.D, -1) if vel.numel() > self.D else vel.reshape(self.D, 1)).expand(self.D, o.numel())
        self.bvel[f][:, o] = v
        self.bflux[f][o] = det * (inv[:, a] * v.T).sum(1)
        self.balpha[f][o] = det * (inv[:, a] ** 2).sum(1)

    # -- operators --
    def fluxes(self, u):
        return [torch.where(self.fixed[f], self.bflux[f],
                            0.5 * ((self.Wn[f] * u[:, self.nb[f]].T).sum(1) + (self.Wc[f >> 1] * u.T).sum(1)))
                for f in range(2 * self.D)]

    def transport(self, u, nu, dirichlet_only=False):
        fl, co = self.fluxes(u), []
        diag = self.det / self.dt
        for f in range(2 * self.D):
            ff = (1.0 if f & 1 else -1.0) * 0.5 * fl[f]
            aP = self.alpha[f >> 1]
            vc = 0.5 * (aP * nu + self.alphaN[f] * (nu if nu.numel() == 1 else nu[self.nb[f]]))
            diag = diag + torch.where(self.fixed[f], 2.0 * nu * aP, ff + vc)
            co.append(torch.where(self.fixed[f], torch.zeros_like(vc), ff - vc))
        return torch.stack([diag] + co) / self.det

    def faces_in(self, nu, value=None):
        """What the prescribed faces add to a transport right-hand side (not yet over det): [components, N]."""
        out = 0.0
        for f in range(2 * self.D):
            v = self.bvel[f] if value is None else value(f)
            out = out + torch.where(self.fixed[f], -v * self.bflux[f] * (1.0 if f & 1 else -1.0)
                                    + v * nu * 2.0 * self.balpha[f], torch.zeros_like(v))
        return out

    def rhs(self, u):
        return u / self.dt + self.faces_in(self.nu) / self.det + self.src

    def pressure(self, A):
        co, ra = [], 1.0 / A
        for f in range(2 * self.D):
            v = 0.5 * (self.alpha[f >> 1] * ra + self.alphaN[f] * ra[self.nb[f]])
            co.append(torch.where(self.fixed[f], torch.zeros_like(v), v))
        return torch.stack([-sum(co)] + co)

    def over(self, C, A, u, us):
        H = sum(C[f + 1] * us[:, self.nb[f]] for f in range(2 * self.D))
        return (u / self.dt - H + self.faces_in(self.nu) / self.det + self.src) / A

    def div(self, h):
        fl = self.fluxes(h)
        return sum(fl[2 * a + 1] - fl[2 * a] for a in range(self.D))

    def correct(self, h, p, A):
        g = []
        for a in range(self.D):
            one = self.fixed[2 * a] | self.fixed[2 * a + 1]
            g.append((p[self.nb[2 * a + 1]] - p[self.nb[2 * a]]) * torch.where(one, 1.0, 0.5).double())
        return h - torch.einsum("in,nij->jn", torch.stack(g), self.Minv) / A

    def mean_free(self, p):
        m = torch.zeros(self.ns, dtype=p.dtype, device=p.device).index_add(0, self.sim, p) / self.count
        return p - m[self.sim]

    # -- systems --
    def mul(self, A, x):
        y = A[0] * x
        for f in range(2 * self.D):
            y = y + A[f + 1] * x[self.nb[f]]
        return y

    def transposed(self, A):
        """The transposed stencil (blocks without connections)."""
        return torch.stack([A[0]] + [torch.where(self.fixed[f], torch.zeros_like(A[0]), A[(f ^ 1) + 1][self.nb[f]])
                                     for f in range(2 * self.D)])

    def cg(self, A, b, x=None, tol=1e-12):
        b = self.mean_free(b)
        x = torch.zeros_like(b) if x is None else x
        r = b - self.mul(A, x)
        stop = tol * float(b.norm())
        z = r / A[0]
        p, rz = z, (r * z).sum()
        for it in range(20000):
            if it % 25 == 0 and not float(r.norm()) > stop:
                break
            q = self.mul(A, p)
            al = rz / (p * q).sum()
            x = x + al * p
            r = r - al * q
            z = r / A[0]
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
        return self.mean_free(x)

    def bicgstab(self, A, b, tol=1e-14):
        x = b / A[0]
        r = b - self.mul(A, x)
        rw, p, rho = r, r, (r * r).sum()
        stop = tol * float(b.norm())
        for _ in range(500):
            if not float(r.norm()) > stop:
                break
            v = self.mul(A, p / A[0])
            al = rho / (rw * v).sum()
            s = r - al * v
            t = self.mul(A, s / A[0])
            om = (t * s).sum() / (t * t).sum()
            x = x + (al * p + om * s) / A[0]
            r = s - om * t
            new = (rw * r).sum()
            p = r + (new / rho) * (al / om) * (p - om * v)
            rho = new
        return x

    def step(self, u, correctors=2):
        C = self.transport(u, self.nu)
        A, b = C[0], self.rhs(u)
        us = torch.stack([_Solve.apply(self, C, b[k], False, None) for k in range(self.D)])
        Pm, p = self.pressure(A), getattr(self, "p", None)
        for _ in range(correctors):
            h = self.over(C, A, u, us)
            p = _Solve.apply(self, Pm, self.div(h), True, None if p is None else p.detach())
            us = self.correct(h, p, A)
        self.p = p.detach()
        return us, p


class _Solve(torch.autograd.Function):
    @staticmethod
    def forward(ctx, flow, A, b, symmetric, guess):
        x = flow.cg(A, b, guess) if symmetric else flow.bicgstab(A, b)
        ctx.flow, ctx.symmetric = flow, symmetric
        ctx.save_for_backward(A, x)
        return x

    @staticmethod
    def backward(ctx, g):
        A, x = ctx.saved_tensors
        fl = ctx.flow
        lam = fl.cg(A, g) if ctx.symmetric else fl.bicgstab(fl.transposed(A), g)
        return None, torch.stack([-lam * x] + [-lam * x[fl.nb[f]] for f in range(2 * fl.D)]), lam, None, None


def _flow(dims, i, nu, dt, faces, source=None):
    one = lambda v: torch.tensor(float(v), dtype=torch.float64, device=_dev())
    return Flow64([dict(coords=i["coords"][0], faces=faces)], one(nu), one(dt), source)


def _flow_batch(c, seed):
    """The batch of a case: largest simulations first, as BatchDomain orders them."""
    bs = _batch_params(c, seed)
    bs = [bs[i] for i in sorted(range(len(bs)), key=lambda i: -bs[i]["u"].numel())]
    wall = torch.zeros(2)
    lid = torch.tensor([1.0, 0.0])
    fl = Flow64([dict(coords=b["coords"][0], faces=[wall, wall, lid, wall]) for b in bs], None, None)
    nu = torch.tensor([b["nu"] for b in bs], dtype=torch.float64, device=_dev())
    fl.dt = torch.tensor([b["dt"] for b in bs], dtype=torch.float64, device=_dev())[fl.sim]
    fl.nu = nu[fl.sim]
    return fl, nu, torch.cat([b["u"].double().reshape(2, -1) for b in bs], dim=1), [b["u"].numel() // 2 for b in bs]


def _packed(x, sizes):
    return torch.cat([t.reshape(-1) for t in x.split(sizes, dim=-1)])


def exact(case, seed):
    c, k = case, case["kind"]
    if k == "gradient":
        fl, nu, u, _ = _flow_batch(c, seed)
        nu, u = nu.requires_grad_(True), u.requires_grad_(True)
        fl.nu, v = nu[fl.sim], u
        for _ in range(c["steps"]):
            v, _p = fl.step(v)
        (0.5 * ((v * v) / (fl.ns * fl.count[fl.sim])).sum()).backward()
        return dict(u=v.detach().reshape(-1), grad_u=u.grad.reshape(-1), grad_nu=nu.grad)
    if k == "forcing":
        i = _inputs(c, seed)
        f = i["f"].reshape(2, -1).clone().requires_grad_(True)
        fl = _flow(2, i, 1e-3, 0.5 / c["n"], [None] * 4, f)
        u, loss, outs = i["u"].reshape(2, -1), 0.0, []
        for s in range(1, c["steps"] + 1):
            u, _p = fl.step(u)
            if s in (c["steps"] // 2, c["steps"]):
                outs.append(u.detach().reshape(-1))
                loss = loss + ((u - i["target"].reshape(2, -1)) ** 2).mean()
        loss.backward()
        return dict(u=outs, grad=f.grad.reshape(-1))
    with torch.no_grad():
        return _exact(c, k, seed)


def _exact(c, k, seed):
    if k == "cavities":
        fl, _nu, u, sizes = _flow_batch(c, seed)
        for _ in range(WARM + c["steps"]):
            u, p = fl.step(u)
        return _packed(u, sizes), p
    if k == "street":
        return _exact_street(c, seed)
    i = _inputs(c, seed)
    wall = torch.zeros(3)
    if k == "channel":
        src = torch.tensor([[1.0], [0.0], [0.0]], dtype=torch.float64, device=_dev())
        fl = _flow(3, i, float(np.float32(1.0 / 180.0)), _channel_dt(c), [None, None, wall, wall, None, None], src)
        u = i["u"].double().reshape(3, -1)
        for _ in range(2 + c["steps"]):
            u, p = fl.step(u)
        return u.reshape(i["u"].shape), p.reshape((1, 1) + i["u"].shape[2:])
    if k == "simulation":
        fl = _flow(3, i, 1e-2, 0.2 / c["n"], [wall, wall, wall, torch.tensor([1.0, 0.0, 0.0]), wall, wall])
        u = i["u"].reshape(3, -1)
        for _ in range(c["steps"]):
            u, p = fl.step(u)
        return u.reshape(i["u"].shape), p.reshape((1, 1) + i["u"].shape[2:])
    if k == "operators":
        w2 = torch.zeros(2)
        fl = _flow(2, i, float(np.float32(1e-3)), float(np.float32(0.5 / c["nx"])), [w2, w2, torch.tensor([1.0, 0.0]), w2])
        u, us, p = i["u"].double().reshape(2, -1), i["us"].double().reshape(2, -1), i["p"].double().reshape(-1)
        C = fl.transport(u, fl.nu)
        A = C[0]
        h = fl.over(C, A, u, us)
        return dict(A=A, C=C, rhs=fl.rhs(u).reshape(-1), P=fl.pressure(A), h=h.reshape(-1), div=fl.div(h),
                    u=fl.correct(h, p, A).reshape(-1), udiv=fl.div(u))
    if k == "skewed":
        return _exact_skewed(c, i)
    if k == "scalars":
        fl = _flow(3, i, float(np.float32(1e-3)), float(np.float32(_scalar_dt(c))), [None, None, wall, wall, None, None])
        u, s = i["u"].double().reshape(3, -1), i["s"].double().reshape(2, -1)
        nu = torch.tensor(float(np.float32(2e-3)), dtype=torch.float64, device=_dev())
        C = fl.transport(u, nu)
        lower = torch.tensor([[1.0], [0.5]], dtype=torch.float64, device=_dev())
        val = lambda f: (lower if f == 2 else torch.zeros_like(lower)).expand(2, fl.N)
        for _ in range(c["steps"]):
            b = s / fl.dt + fl.faces_in(nu, val) / fl.det
            s = torch.stack([fl.bicgstab(C, b[j]) for j in range(2)])
        g = []
        for a in range(3):
            lo, hi = [torch.where(fl.fixed[f], fl.bvel[f], u[:, fl.nb[f]]) for f in (2 * a, 2 * a + 1)]
            g.append((hi - lo) / (2.0 - 0.5 * fl.fixed[2 * a].double() - 0.5 * fl.fixed[2 * a + 1].double()))
        G = torch.einsum("kcn,nkj->ncj", torch.stack(g), fl.Minv)
        S = 0.5 * (G + G.transpose(1, 2))
        sg = 0.17 ** 2 * (fl.M ** 2).sum(1).max(1).values * (2.0 * (S * S).sum((1, 2))).sqrt()
        return dict(s=s.reshape(i["s"].shape), nu=[sg.reshape((1, 1) + i["u"].shape[2:])])
    return _exact_padding(c, i)


def _exact_skewed(c, i):
    """Fully periodic, so a corner value is the mean of its four cells: the direct matrix flag takes the two face
    neighbours, the centre flag the cell itself and the diagonal flag leaves the fourth to the right-hand side."""
    D, dev = 3, _dev()
    fl = _flow(3, i, 1e-3, 0.5 / c["nx"], [None] * 6)
    u, p = i["u"].reshape(3, -1), i["p"].reshape(-1)
    full = fl.det[:, None, None] * fl.Minv @ fl.Minv.transpose(1, 2)

    def tangential(w):
        """Per face and tangential axis: face-averaged off-diagonal coefficient, weighted by w per cell."""
        return {(f, t): 0.5 * (full[:, f >> 1, t] * w + full[fl.nb[f], f >> 1, t] * w[fl.nb[f]])
                for f in range(6) for t in range(3) if t != f >> 1}

    def terms(fa, sign):
        add = torch.zeros((7, fl.N), dtype=torch.float64, device=dev)
        for (f, t), a in fa.items():
            for g in (2 * t, 2 * t + 1):  # the cell's and the face neighbour's share cancel between the two corners
                add[g + 1] += sign * (1.0 if f & 1 else -1.0) * (1.0 if g & 1 else -1.0) * a / 4
        return add

    def explicit(fa, x):
        s = 0.0
        for (f, t), a in fa.items():
            for g in (2 * t, 2 * t + 1):
                s = s - (1.0 if f & 1 else -1.0) * (1.0 if g & 1 else -1.0) * a * x[..., fl.nb[g][fl.nb[f]]] / 4
        return s

    fv = tangential(torch.full((fl.N,), 1e-3, dtype=torch.float64, device=dev))
    C = fl.transport(u, fl.nu) + terms(fv, -1.0) / fl.det
    A = C[0]
    fp = tangential(1.0 / A)
    h = fl.over(C, A, u, u)
    return dict(A=A, C=C, rhs=(fl.rhs(u) - explicit(fv, u) / fl.det).reshape(-1), P=fl.pressure(A) + terms(fp, 1.0),
                h=h.reshape(-1), div=fl.div(h) + explicit(fp, p))


def _exact_street(c, seed):
    spec = _street_spec(c, seed)
    f32 = lambda a: torch.as_tensor(np.asarray(a)).float().double().to(_dev())
    faces = [[torch.zeros(2) for _ in range(4)] for _ in spec["blocks"]]
    fid = {"-x": 0, "+x": 1, "-y": 2, "+y": 3}
    for op in spec["ops"]:
        if op[0] == "connect":
            b1, f1, b2, f2, ax = op[1], fid[op[2]], op[3], fid[op[4]], fid[op[5]]
            faces[b1][f1], faces[b2][f2] = (b2, f2, ax & 1), (b1, f1, ax & 1)
        elif op[0] == "close":
            faces[op[1]][fid[op[2]]] = f32(op[3]).reshape(2, -1).squeeze(-1)
    one = lambda v: torch.tensor(float(np.float32(v)), dtype=torch.float64, device=_dev())
    fl = Flow64([dict(coords=f32(b["coords"][0]), faces=fc) for b, fc in zip(spec["blocks"], faces)],
                one(spec["viscosity"]), one(TIME_STEP))
    u = torch.cat([f32(b["velocity"]).reshape(2, -1) for b in spec["blocks"]], dim=1)
    (ob, of), = spec["outflow"]
    cells, M = fl.bfaces[(ob, of)]
    out = faces[ob][of].to(_dev())
    speed = torch.linalg.inv(M)[:, of >> 1, 0]  # characteristic velocity (1, 0) through the face
    sign = torch.tensor([1.0 if f & 1 else -1.0 for f in range(4)], dtype=torch.float64, device=_dev())
    for _ in range(2 + c["steps"]):
        out = out - (1.0 - 1.0 / (1.0 + 2.0 * fl.dt * speed)) * (out - u[:, cells])
        fl.set_face(ob, of, out)
        free = fl.bflux[of][cells].sum()
        total = (fl.bflux.sum(1) * sign).sum()
        if abs(float(total)) > 1e-7:
            out = out * (-(total - free) / free)
            fl.set_face(ob, of, out)
        u, p = fl.step(u)
    return dict(u=u, p=p, out=out.reshape(1, 2, -1, 1))


def _exact_padding(c, i):
    m, q = c["m"], c["kernel"] // 2
    x = [t.double().requires_grad_(True) for t in i["x"]]
    with torch.enable_grad():
        whole = torch.cat([torch.cat([x[0], x[1]], 3), torch.cat([x[2], x[3]], 3)], 2)
        whole = torch.nn.functional.pad(whole, (q, q, q, q))
        y = []
        for b, (h, w) in enumerate(_padding_sizes(m)):
            y0, x0 = (b // 2) * m, (b % 2) * m
            y.append(whole[:, :, y0:y0 + h + 2 * q, x0:x0 + w + 2 * q])
        torch.autograd.backward(y, [t.double() for t in i["g"]])
    return dict(y=[t.detach() for t in y], grad=[t.grad for t in x])

