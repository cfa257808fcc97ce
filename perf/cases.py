"""The work that users of the NuSiF library have it do, as cases to be measured.

Kinds of case, each through the package's public entry points:

  rb       one red-black SOR pressure solve, the reference's own solver
  mg       one multigrid pressure solve (solver mg or mg-mixed)
  predict  the first half of a time step: CFL step size, boundary conditions,
           F/G/H and the right-hand side of the pressure equation
  step     one whole time step of a running simulation
  batch    one time step of several uneven cavities advanced together
  forward  the U-Net of the learned warm start on a feature volume
  train    one training step of that network

A solve starts every pass from the same earlier pressure, as the solve of one
time step does; a step, a batch and a training step advance their state.
"""
import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch
import torch.nn.functional as nnf

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT / "cfd-bench_gb300"))

import nusif  # noqa: E402
from nusif import abi, learn, params  # noqa: E402

WEIGHTS = ROOT / "cfd-bench_gb300" / "nusif" / "weights" / "unet_cavity128.npz"


def _box(n, length=(1.0, 1.0, 1.0)):
    return {"nx": n[0], "ny": n[1], "nz": n[2], "lx": length[0], "ly": length[1], "lz": length[2]}


def listed():
    return [
        # the plain method's CPU-size configuration: 64^3 cavity, omega 1.7, eps 1e-3, itermax 500
        {"name": "rb_cavity64", "kind": "rb", **_box((64, 64, 64)), "omg": 1.7, "eps": 1e-3,
         "itermax": 500, "arith": "df32"},
        # the reference's canal.par: a 30 x 4 x 4 duct of 200 x 40 x 40 cells, eps 1e-4, itermax 500
        {"name": "rb_canal200", "kind": "rb", **_box((200, 40, 40), (30.0, 4.0, 4.0)), "omg": 1.8,
         "eps": 1e-4, "itermax": 500, "arith": "df32"},
        # the reference's dcavity.par: 128^3, omega 1.8, eps 1e-3, itermax 1000
        {"name": "rb_cavity128", "kind": "rb", **_box((128, 128, 128)), "omg": 1.8, "eps": 1e-3,
         "itermax": 1000, "arith": "df32"},
        # plain FP64 multigrid, V(2,2) Gauss-Seidel cycles to 1e-6
        {"name": "mg_cavity128", "kind": "mg", **_box((128, 128, 128)), "solver": "mg", "pre": 2,
         "post": 2, "omega": 1.0, "rtol": 1e-6, "arith": "df32"},
        # mixed-precision multigrid on the channel, to 1e-8
        {"name": "mixed_channel512", "kind": "mg", **_box((512, 128, 128), (4.0, 1.0, 1.0)),
         "solver": "mg-mixed", "pre": 2, "post": 2, "omega": 1.0, "rtol": 1e-8, "arith": "df32"},
        # mixed-precision multigrid on a grid with axes that stop halving early
        {"name": "mixed_ragged", "kind": "mg", **_box((72, 36, 60), (2.0, 1.0, 1.5)),
         "solver": "mg-mixed", "pre": 1, "post": 1, "omega": 1.3, "rtol": 1e-6, "arith": "df32"},
        # the predictor half of a step on the channel with inflow and outflow
        {"name": "predict_channel512", "kind": "predict", **_box((512, 128, 128), (4.0, 1.0, 1.0)),
         "flow": "canal", "re": 100.0, "grav": 0.0, "arith": "df32"},
        # a whole step of the smallest useful cavity with the reference's solver: launches and latency
        {"name": "step_cavity16", "kind": "step", **_box((16, 16, 16)), "flow": "dcavity",
         "re": 1000.0, "solver": "rb", "pre": 2, "post": 2, "omega": 1.0, "guess": "previous",
         "fuse_dt": 0},
        # a whole step of the 256^3 cavity with the fastest solver (without the network)
        {"name": "step_cavity256", "kind": "step", **_box((256, 256, 256)), "flow": "dcavity",
         "re": 1000.0, "solver": "mg-mixed", "pre": 1, "post": 1, "omega": 1.3,
         "guess": "quadratic", "fuse_dt": 1},
        # uneven cavities of a parameter study, one graph launch per step
        {"name": "batch_uneven", "kind": "batch", "edges": "32,128,48,64,96,32,64,48,96,64,32,48"},
        # the network on the half-resolution grid of a 256^3 simulation
        {"name": "unet_forward128", "kind": "forward", "b": 1, "z": 128, "y": 128, "x": 128},
        # a training batch of eight pairs recorded at 128^3
        {"name": "unet_train64", "kind": "train", "b": 8, "z": 64, "y": 64, "x": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _axes(rng, lo, hi, cells, step=1):
    """Three axis lengths, log-uniform, multiples of `step`, at most `cells` cells in all."""
    while True:
        n = [max(lo, _log(rng, lo, hi) // step * step) for _ in range(3)]
        if n[0] * n[1] * n[2] <= cells:
            return n


# multigrid halves even axes: grids of odd or barely even axes are left to small sizes
MG_CELLS = {1: 32 ** 3, 4: 96 ** 3, 8: 160 ** 3, 16: 192 ** 3}


def draw(rng):
    kind = rng.choice(["rb", "rb", "rb", "mg", "mg", "mg", "predict", "predict", "step", "step",
                       "batch", "forward", "train"])
    length = [rng.choice([1.0, 1.0, 1.5, 2.0, 4.0]) for _ in range(3)]
    if kind == "rb":
        n = _axes(rng, 6, 160, 128 ** 3)
        return {"kind": "rb", **_box(n, length), "omg": rng.choice([1.7, 1.8]),
                "eps": rng.choice([1e-3, 1e-4]), "itermax": rng.choice([100, 200, 500, 1000]),
                "arith": rng.choice(["df32", "df32", "df32", "fp64"])}
    if kind == "mg":
        solver = rng.choice(["mg", "mg-mixed", "mg-mixed"])
        step = rng.choice([1, 4, 8, 8, 16, 16])
        n = _axes(rng, 16, 320, min(MG_CELLS[step], 128 ** 3 if solver == "mg" else 192 ** 3), step)
        pre, omega = rng.choice([(1, 1.3), (2, 1.0), (2, 1.3)])
        return {"kind": "mg", **_box(n, [x / max(n) for x in n]), "solver": solver,
                "pre": pre, "post": pre, "omega": omega, "rtol": rng.choice([1e-6, 1e-8]),
                "arith": rng.choice(["df32", "df32", "df32", "fp64"])}
    if kind == "predict":
        n = _axes(rng, 8, 384, 192 ** 3)
        return {"kind": "predict", **_box(n, length), "flow": rng.choice(["dcavity", "canal"]),
                "re": rng.choice([100.0, 1000.0]), "grav": rng.choice([0.0, 0.0, -0.1]),
                "arith": rng.choice(["df32", "df32", "df32", "fp64"])}
    if kind == "step":
        solver = rng.choice(["rb", "mg-mixed", "mg-mixed"])
        step = 1 if solver == "rb" else rng.choice([4, 8, 8, 16])
        n = _axes(rng, 8, 48, 48 ** 3) if step == 1 else _axes(rng, 16, 256, MG_CELLS[step], step)
        pre, omega = rng.choice([(1, 1.3), (2, 1.0)])
        return {"kind": "step", **_box(n, [x / max(n) for x in n]),
                "flow": rng.choice(["dcavity", "dcavity", "canal"]),
                "re": rng.choice([100.0, 1000.0, 5000.0]), "solver": solver, "pre": pre,
                "post": pre, "omega": omega,
                "guess": rng.choice(["previous", "extrapolate", "quadratic"]),
                "fuse_dt": rng.choice([0, 1])}
    if kind == "batch":
        edges = [rng.choice([32, 48, 64, 96]) for _ in range(rng.randint(2, 12))]
        return {"kind": "batch", "edges": ",".join(map(str, edges))}
    z, y, x = (4 * max(2, _log(rng, 2, 32)) for _ in range(3))
    if kind == "forward":
        return {"kind": "forward", "b": rng.choice([1, 1, 2]) if z * y * x <= 64 ** 3 else 1,
                "z": z, "y": y, "x": x}
    z, y, x = (min(64, e) for e in (z, y, x))
    return {"kind": "train", "b": rng.randint(1, 8), "z": z, "y": y, "x": x}


# ---- inputs -------------------------------------------------------------------------------


def _n(case):
    return case["nx"], case["ny"], case["nz"]


def _len(case):
    return case["lx"], case["ly"], case["lz"]


def _pressure(case, rng, modes=10):
    """A smooth pressure with zero normal gradient at the walls, interior cells only."""
    axes = []
    for n in _n(case):
        axes.append((torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) * (math.pi / n))
    p = torch.zeros(_n(case)[::-1], dtype=torch.float64, device="cuda")
    for _ in range(modes):
        m = rng.integers(0, 5, 3)
        if not m.any():
            m[0] = 1
        x, y, z = (torch.cos(float(k) * a) for k, a in zip(m, axes))
        amp = rng.standard_normal() / (1.0 + float((m ** 2).sum()))
        p += amp * z[:, None, None] * y[None, :, None] * x[None, None, :]
    return p


def _neumann_pad(p):
    """The padded array: wall ghosts copy their cell, edges and corners are zero."""
    out = torch.zeros([s + 2 for s in p.shape], dtype=p.dtype, device=p.device)
    out[1:-1, 1:-1, 1:-1] = p
    _ghosts(out)
    return out


def _ghosts(p):
    c = slice(1, -1)
    p[0, c, c], p[-1, c, c] = p[1, c, c], p[-2, c, c]
    p[c, 0, c], p[c, -1, c] = p[c, 1, c], p[c, -2, c]
    p[c, c, 0], p[c, c, -1] = p[c, c, 1], p[c, c, -2]


def _lap(p, ih2):
    c, lo, hi = slice(1, -1), slice(0, -2), slice(2, None)
    q = p[c, c, c]
    return ((p[c, c, hi] - 2.0 * q + p[c, c, lo]) * ih2[0] +
            (p[c, hi, c] - 2.0 * q + p[c, lo, c]) * ih2[1] +
            (p[hi, c, c] - 2.0 * q + p[lo, c, c]) * ih2[2])


def _poisson(case, seed):
    """An earlier pressure and the right-hand side of a later one some per cent away from it,
    with the cell-scale noise that the velocities' divergence carries (padded arrays)."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    ih2 = [(n / x) ** 2 for n, x in zip(_n(case), _len(case))]
    p0 = _pressure(case, rng)
    noise = torch.randn(p0.shape, dtype=torch.float64, device="cuda", generator=gen)
    p1 = p0 + 0.03 * _pressure(case, rng) + 1e-4 * noise
    rhs = torch.zeros([s + 2 for s in p0.shape], dtype=torch.float64, device="cuda")
    rhs[1:-1, 1:-1, 1:-1] = _lap(_neumann_pad(p1), ih2)
    return _neumann_pad(p0), rhs


def _velocity(case, seed):
    """A divergence-free staggered velocity of size 1 without flow through the walls (plus a
    uniform stream in a canal), padded arrays."""
    rng = np.random.default_rng(seed)
    n, length = _n(case), _len(case)
    face, centre = [], []
    for m in n:
        q = torch.arange(m + 2, dtype=torch.float64, device="cuda")
        face.append(q * (math.pi / m))
        centre.append((q - 0.5) * (math.pi / m))
    vel = [torch.zeros([m + 2 for m in n[::-1]], dtype=torch.float64, device="cuda")
           for _ in range(3)]
    for _ in range(6):
        m = rng.integers(1, 5, 3)
        a = rng.standard_normal(3) / float(m.sum())
        a[2] = -(a[0] * m[0] / length[0] + a[1] * m[1] / length[1]) * length[2] / m[2]
        for c in range(3):
            f = [torch.sin(float(m[d]) * face[d]) if d == c else torch.cos(float(m[d]) * centre[d])
                 for d in range(3)]
            vel[c] += float(a[c]) * f[2][:, None, None] * f[1][None, :, None] * f[0][None, None, :]
    top = max(float(q.abs().max()) for q in vel)
    for q in vel:
        q /= top
    if case["flow"] == "canal":
        for q in vel:
            q *= 0.3
        vel[0] += 1.0
    return vel


def _par(case):
    """The .par values of a case."""
    (i, j, k), (x, y, z) = _n(case), _len(case)
    par = dict(params.CANAL if case.get("flow") == "canal" else params.DCAVITY, imax=i, jmax=j,
               kmax=k, xlength=x, ylength=y, zlength=z, te=1e9, tau=0.5, re=case.get("re", 1000.0),
               gx=case.get("grav", 0.0), gy=0.0, gz=case.get("grav", 0.0),
               omg=case.get("omg", 1.7), eps=case.get("eps", 1e-3),
               itermax=case.get("itermax", 500), solver=case.get("solver", "rb"),
               rtol=case.get("rtol", 1e-6), arith=case.get("arith", "df32"),
               fuse_dt=case.get("fuse_dt", 0), u_init=0.0)
    if par["name"] == "canal":
        par["inflow"] = 1.0
    if "pre" in case:
        par.update(mg_pre=case["pre"], mg_post=case["post"], mg_omega=case["omega"])
    if "guess" in case:
        par["mg_guess"] = case["guess"]
    return par


class _Owner:
    """Closes a batch or a network with its last user."""

    def __init__(self, held):
        self.held = held

    def __del__(self):
        self.held.close()


class _Field:
    """A field of the library as torch sees it: the library's own device memory, which lives as
    long as the simulation or batch that owns it (a tensor made from this keeps it alive)."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {
            "shape": tuple(shape), "typestr": "<f8", "version": 3,
            "data": (ctypes.cast(ptr, ctypes.c_void_p).value, False)}


def _view(d, name, owner):
    g = d.grid
    shape = (g.kmax + 2, g.jmax + 2, g.imax + 2)
    return torch.as_tensor(_Field(getattr(d, name), shape, owner), device="cuda")


def _features(case, seed):
    """Feature volumes as the solver makes them: a residual and a right-hand side of RMS 1."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    b, z, y, x = case["b"], case["z"], case["y"], case["x"]
    small = torch.randn((b, 2, max(2, z // 8), max(2, y // 8), max(2, x // 8)), device="cuda",
                        generator=gen)
    f = nnf.interpolate(small, size=(z, y, x), mode="trilinear", align_corners=False)
    f += 0.3 * torch.randn(f.shape, device="cuda", generator=gen)
    f /= f.square().mean(dim=(2, 3, 4), keepdim=True).sqrt()
    target = 0.1 * f[:, 0] + 0.05 * torch.randn((b, z, y, x), device="cuda", generator=gen)
    return f.permute(0, 2, 3, 4, 1).contiguous(), target.contiguous()


# 3-level U-Net: name, input channels, output channels
LAYERS = [("e0a", 2, 16), ("e0b", 16, 16), ("e1a", 16, 32), ("e1b", 32, 32), ("e2a", 32, 64),
          ("d1a", 96, 32), ("d1b", 32, 32), ("d0a", 48, 16), ("d0b", 16, 16), ("out", 16, 1)]


def _start_weights(seed):
    """He-normal weights and small biases, the flat layout of the network's parameters."""
    rng = np.random.default_rng(seed)
    parts = []
    for _, ci, co in LAYERS:
        parts.append(rng.standard_normal(27 * co * ci) * math.sqrt(2.0 / (27 * ci)))
        parts.append(0.01 * rng.standard_normal(co))
    return np.concatenate(parts).astype(np.float32)


def _batch_cases(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for n in map(int, case["edges"].split(",")):
        out.append({"kind": "step", **_box((n, n, n)), "flow": "dcavity",
                    "re": float(rng.uniform(100.0, 5000.0)), "solver": "mg-mixed", "pre": 1,
                    "post": 1, "omega": 1.3, "guess": "quadratic"})
    return out


class State:
    pass


def prepare(case, seed):
    st = State()
    st.kind = kind = case["kind"]
    if kind in ("rb", "mg"):
        st.sim = nusif.Simulation(_par(case))
        st.p0, rhs = _poisson(case, seed)
        st.sim.set_field("rhs", rhs.cpu().numpy())
        st.p = _view(st.sim.d, "p", st.sim)
    elif kind in ("predict", "step"):
        st.sim = nusif.Simulation(_par(case))
        for name, q in zip("uvw", _velocity(case, seed)):
            st.sim.set_field(name, q.cpu().numpy())
        names = "uvwfgh" if kind == "predict" else "uvwp"
        st.out = {name: _view(st.sim.d, name, st.sim) for name in names}
        if kind == "predict":
            st.out["rhs"] = _view(st.sim.d, "rhs", st.sim)
    elif kind == "batch":
        cases = _batch_cases(case, seed)
        st.batch = nusif.Batch([_par(c) for c in cases])
        st.owner = _Owner(st.batch)
        st.out = []
        for q, c in enumerate(cases):
            d = ctypes.POINTER(abi.Discretization)()
            st.batch.lib.nusifBatchInstance(st.batch.handle, q, ctypes.byref(d), None)
            for f, a in zip("uvw", _velocity(c, seed + q)):
                host = np.ascontiguousarray(a.cpu().numpy())
                st.batch.lib.nusifUploadField(d, abi.FIELD_INDEX[f],
                                              host.ctypes.data_as(abi.c_double_p))
            abi.check(st.batch.lib)
            st.out.append({name: _view(d.contents, name, st.owner) for name in "uvwp"})
    elif kind == "forward":
        st.net = learn.load_net(WEIGHTS)
        st.owner = _Owner(st.net)
        st.x, _ = _features(case, seed)
    else:
        st.net = nusif.UNet(seed=0)
        st.owner = _Owner(st.net)
        st.net.set_params(_start_weights(seed))
        st.x, st.t = _features(case, seed)
    return st


def run(st):
    if st.kind in ("rb", "mg"):
        st.p.copy_(st.p0)
        st.sim.solve()
        return {"p": st.p, "iterations": st.sim.iterations}
    if st.kind == "predict":
        sim = st.sim
        sim.compute_timestep()
        sim.set_boundary_conditions()
        sim.set_special_boundary_condition()
        sim.compute_fg()
        sim.compute_rhs()
        return {"dt": sim.dt, **st.out}
    if st.kind == "step":
        info = st.sim.step()
        return {"dt": info.dt, "iterations": info.it, **st.out}
    if st.kind == "batch":
        st.batch.step()
        return st.out
    if st.kind == "forward":
        return st.net.forward(st.x)
    # a late iteration of a decaying schedule: Adam's first steps move each weight by about lr
    loss = st.net.train_step(st.x, st.t, lr=1e-5)
    return {"loss": loss, "grads": st.net.grads(), "params": st.net.params()}


# ---- what a pass cannot do without ----------------------------------------------------------


def _net_flops(cells):
    """Multiply-adds of the forward convolutions, times two."""
    level = {"e0a": 1, "e0b": 1, "e1a": 8, "e1b": 8, "e2a": 64, "d1a": 8, "d1b": 8, "d0a": 1,
             "d0b": 1, "out": 1}
    return sum(2.0 * 27 * ci * co * cells / level[name] for name, ci, co in LAYERS)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        cells = sum(int(n) ** 3 for n in case["edges"].split(","))
    elif kind in ("forward", "train"):
        cells = case["b"] * case["z"] * case["y"] * case["x"]
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "rb":  # p and rhs in, p out; 15 operations per cell and iteration, half of itermax
        return {"bytes": 24.0 * cells, "flops": 15.0 * cells * case["itermax"] / 2}
    if kind == "mg":  # p and rhs in, p out; about four V-cycles
        sweeps = (case["pre"] + case["post"] + 2) * 8 / 7
        return {"bytes": 24.0 * cells, "flops": 4 * 15.0 * sweeps * cells}
    if kind == "predict":  # u, v, w in; f, g, h, rhs out
        return {"bytes": 56.0 * cells, "flops": 160.0 * cells}
    if kind in ("step", "batch"):  # u, v, w, p in and out
        return {"bytes": 64.0 * cells, "flops": 500.0 * cells}
    if kind == "forward":  # two features in, one value out
        return {"bytes": 12.0 * cells, "flops": _net_flops(cells)}
    return {"bytes": 12.0 * cells, "flops": 3 * _net_flops(cells)}


# ---- the same outputs in 64 bits ------------------------------------------------------------


def _exact_rb(case, seed):
    p, rhs = _poisson(case, seed)
    n, ih2 = _n(case), [(m / x) ** 2 for m, x in zip(_n(case), _len(case))]
    h2 = [(x / m) ** 2 for m, x in zip(n, _len(case))]
    factor = (case["omg"] * 0.5 * h2[0] * h2[1] * h2[2] /
              (h2[1] * h2[2] + h2[0] * h2[2] + h2[0] * h2[1]))
    i, j, k = (torch.arange(m, device="cuda") for m in n)
    parity = (k[:, None, None] + j[None, :, None] + i[None, None, :] + 1) % 2  # of 1-based i+j+k
    masks = [(parity == 1).double(), (parity == 0).double()]
    inner, b = p[1:-1, 1:-1, 1:-1], rhs[1:-1, 1:-1, 1:-1]
    res, it, cells = 1.0, 0, n[0] * n[1] * n[2]
    while res >= case["eps"] ** 2 and it < case["itermax"]:
        total = 0.0
        for m in masks:
            r = (b - _lap(p, ih2)) * m
            inner -= factor * r
            total = total + r.square().sum()
        _ghosts(p)
        res = (res + float(total)) / cells
        it += 1
    return {"p": p, "iterations": None}


def _boundaries(case, u, v, w):
    """No-slip walls (outflow at both x-ends of a canal), then the lid or the inflow."""
    vel, c = (u, v, w), slice(1, -1)
    for axis, high in ((1, 1), (1, 0), (0, 0), (0, 1), (2, 0), (2, 1)):
        dim = 2 - axis  # arrays are [k][j][i]
        n = u.shape[dim] - 2
        out = case["flow"] == "canal" and axis == 0

        def at(q):
            s = [c, c, c]
            s[dim] = q
            return tuple(s)

        for comp in range(3):
            q = vel[comp]
            if comp == axis:
                q[at(n if high else 0)] = q[at(n - 1 if high else 1)] if out else 0.0
            else:
                inside = q[at(n if high else 1)]
                q[at(n + 1 if high else 0)] = inside if out else -inside
    if case["flow"] == "canal":
        u[1:-1, 1:-1, 0] = 1.0
    else:
        u[1:-2, -1, 1:-2] = 2.0 - u[1:-2, -2, 1:-2]


def _exact_predict(case, seed):
    u, v, w = _velocity(case, seed)
    n, length = _n(case), _len(case)
    h = [x / m for m, x in zip(n, length)]
    dt = 0.5 * case["re"] / sum(1.0 / q ** 2 for q in h)
    for q, s in zip((u, v, w), h):
        dt = min(dt, s / float(q.abs().max()))
    dt *= 0.5
    _boundaries(case, u, v, w)
    gamma, ire = 0.9, 1.0 / case["re"]

    def sh(q, di=0, dj=0, dk=0):
        return q[1 + dk:q.shape[0] - 1 + dk, 1 + dj:q.shape[1] - 1 + dj, 1 + di:q.shape[2] - 1 + di]

    step = [{"di": 1}, {"dj": 1}, {"dk": 1}]

    def off(*ds):
        o = {"di": 0, "dj": 0, "dk": 0}
        for d, s in ds:
            o["d" + "ijk"[d]] += s
        return o

    vel, out = (u, v, w), []
    for c in range(3):
        q = vel[c]
        q0 = sh(q)
        total = torch.zeros_like(q0)
        for d in range(3):
            up, dn = sh(q, **off((d, 1))), sh(q, **off((d, -1)))
            total += ire / h[d] ** 2 * (up - 2.0 * q0 + dn)
            t = vel[d]
            cp = sh(t) + sh(t, **off((c, 1)))
            cm = sh(t, **off((d, -1))) + sh(t, **off((d, -1), (c, 1)))
            if c == 1 and d == 2:
                dn = up  # the reference's z-convection of v reads the upper neighbour twice
            total -= 0.25 / h[d] * (cp * (q0 + up) - cm * (q0 + dn))
            total -= gamma * 0.25 / h[d] * (cp.abs() * (q0 - up) + cm.abs() * (q0 - dn))
        g = case["grav"] if c != 1 else 0.0
        f = torch.zeros_like(q)
        f[1:-1, 1:-1, 1:-1] = q0 + dt * (total + g)
        lo, hi = [slice(1, -1)] * 3, [slice(1, -1)] * 3
        lo[2 - c], hi[2 - c] = 0, n[c]
        f[tuple(lo)], f[tuple(hi)] = q[tuple(lo)], q[tuple(hi)]
        out.append(f)
    rhs = torch.zeros_like(u)
    rhs[1:-1, 1:-1, 1:-1] = sum((sh(f) - sh(f, **{k: -s for k, s in step[c].items()})) / h[c]
                                for c, f in enumerate(out)) / dt
    return {"dt": dt, "u": u, "v": v, "w": w, "f": out[0], "g": out[1], "h": out[2], "rhs": rhs}


def _network(flat, x):
    """The U-Net in 64 bits on x [B][Z][Y][X][2]; flat: its parameters."""
    p, o = {}, 0
    for name, ci, co in LAYERS:
        wt = flat[o:o + 27 * co * ci].reshape(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2)
        o += 27 * co * ci
        p[name] = (wt, flat[o:o + co])
        o += co

    def conv(name, q):
        r = nnf.conv3d(q, *p[name], padding=1)
        return r if name == "out" else nnf.relu(r)

    def up(q):
        return nnf.interpolate(q, scale_factor=2, mode="nearest")

    e0 = conv("e0b", conv("e0a", x.permute(0, 4, 1, 2, 3)))
    e1 = conv("e1b", conv("e1a", nnf.avg_pool3d(e0, 2)))
    e2 = conv("e2a", nnf.avg_pool3d(e1, 2))
    d1 = conv("d1b", conv("d1a", torch.cat([up(e2), e1], 1)))
    d0 = conv("d0b", conv("d0a", torch.cat([up(d1), e0], 1)))
    return conv("out", d0)[:, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "rb":
        return _exact_rb(case, seed)
    if kind == "predict":
        return _exact_predict(case, seed)
    if kind == "forward":
        x, _ = _features(case, seed)
        flat = torch.from_numpy(np.load(WEIGHTS)["params"]).cuda().double()
        with torch.no_grad():
            return _network(flat, x.double())
    if kind == "train":
        x, t = _features(case, seed)
        flat = torch.from_numpy(_start_weights(seed)).cuda().double().requires_grad_()
        loss = 0.0
        for b in range(x.shape[0]):  # one volume at a time: the graph of a batch is large
            part = (_network(flat, x[b:b + 1].double()) - t[b:b + 1].double()).square().sum()
            part = part / t.numel()
            part.backward()
            loss += float(part)
        return {"loss": loss, "grads": flat.grad.detach(), "params": None}
    return None
