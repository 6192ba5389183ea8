"""Performance cases of the Poisson library: what its users have it do, through its public entry points.

A model run calls solve_poisson! twice per time step on one grid for thousands of steps, or the whole implicit half
step around it; an ensemble driver solves many members together; the learned warm start is applied to a field and
trained.  The cases take these calls from the periodic hill (40 x 1 x 40, latency only) to the 512 x 512 x 192
domain, with the inputs of the seeded workloads (configs.py): isolated mountains, hills and ridges on stretched or
uniform terrain-following grids, white-noise or wave-packet right-hand sides, tolerance 1e-10 on the true residual.

prepare() makes every input on the GPU from the seed; exact() repeats the call in FP64 with plain torch.  In exact()
the operator is never assembled: A q = -div(correction(q)), the identity that makes the corrected winds
divergence-free (compute_lhs!.jl:68-160 of what correct!.jl:164-385 subtracts), solved by BiCGSTAB
preconditioned with the horizontally averaged operator.
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "pincflow.jl_b200"))

import pincflow_poisson as pcf  # noqa: E402
from pincflow_poisson import configs, learned  # noqa: E402
from pincflow_poisson.fields import Domain, constants  # noqa: E402

H = 3  # halo width of every haloed field (the reference's nbx = nby = nbz)
F64 = torch.float64
DEV = "cuda"


def listed():
    fast = dict(kind="solve", precision="mixed", multigrid=True)
    return [
        # the periodic-hill example: host arrays, 1,600 cells, reference arithmetic
        dict(name="hill", kind="solve", terrain="hill", nx=40, ny=1, nz=40, precision="fp64", multigrid=False, host=True),
        # the solver as configured for speed, from the smallest ensemble grid to the largest domain
        dict(name="solve_64x64x32", terrain="hills", nx=64, ny=64, nz=32, host=False, **fast),
        dict(name="solve_150x90x45", terrain="mountain", nx=150, ny=90, nz=45, host=False, **fast),
        dict(name="solve_128x128x64", terrain="hills", nx=128, ny=128, nz=64, host=False, **fast),
        dict(name="solve_256x256x128", terrain="mountain", nx=256, ny=256, nz=128, host=False, **fast),
        dict(name="solve_512x512x192", terrain="ridges", nx=512, ny=512, nz=192, host=False, **fast),
        # the reference's own algorithm: FP64 throughout, line-relaxation preconditioner
        dict(name="reference_96x96x48", kind="solve", terrain="hills", nx=96, ny=96, nz=48, precision="fp64",
             multigrid=False, host=False),
        # FP32 inner iteration with the reference's preconditioner
        dict(name="mixed_128x96x48", kind="solve", terrain="mountain", nx=128, ny=96, nz=48, precision="mixed",
             multigrid=False, host=False),
        # 32 uneven members solved together
        dict(name="ensemble_32", kind="ensemble", members=32, sizes="64,96,128,192"),
        # the implicit half step around the solve: predictor, divergence, solve, corrector
        dict(name="step_256x256x128", kind="step", terrain="mountain", nx=256, ny=256, nz=128),
        # the implicit predictor alone: Compressible, wave forcing, damping on all faces
        dict(name="predictor_192x160x96", kind="predictor", terrain="mountain", nx=192, ny=160, nz=96),
        # the learned warm start: one application to a field, and loss and gradients of one training sample
        dict(name="network_128x128x64", kind="network", nx=128, ny=128, nz=64),
    ]


def _size(rng, lo, hi):
    """An extent spread over the logarithm of [lo, hi]: mostly multiples of 8, sometimes any number."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n if rng.random() < 0.25 else max(8, n // 8 * 8)


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "reference", "mixed", "ensemble", "step", "predictor", "network"])
    if kind == "ensemble":
        sizes = sorted(rng.sample(range(32, 161, 8), 3))
        return dict(kind=kind, members=rng.randint(3, 16), sizes=",".join(str(s) for s in sizes))
    if kind == "network":
        return dict(kind=kind, nx=_size(rng, 24, 200), ny=_size(rng, 24, 200), nz=rng.randint(32, 128))
    terrain = rng.choice(["hills", "mountain", "ridges"])
    if kind in ("reference", "mixed"):
        # these take hundreds of iterations: moderate grids
        return dict(kind="solve", terrain=terrain, nx=_size(rng, 24, 128), ny=_size(rng, 24, 128), nz=rng.randint(16, 64),
                    precision="fp64" if kind == "reference" else "mixed", multigrid=False, host=rng.random() < 0.3)
    nx, ny, nz = _size(rng, 32, 384), _size(rng, 32, 384), rng.randint(16, 128)
    while (nx % 8 or ny % 8) and nx * ny * nz > 1_000_000:  # ragged grids stay moderate
        nx, ny, nz = max(33, nx // 2), max(33, ny // 2), max(16, nz // 2)
    case = dict(kind=kind, terrain=terrain, nx=nx, ny=ny, nz=nz)
    if kind == "solve":
        case.update(precision="mixed", multigrid=True, host=nx * ny * nz < 200_000 and rng.random() < 0.5)
    return case


# ------------------------------------------------------------------ inputs --


class Box:
    """A grid and its state: views of haloed fields, indexed [k, j, i]."""

    def __init__(self, nx, ny, nz):
        self.nx, self.ny, self.nz = nx, ny, nz
        self.shape = (nz + 2 * H, ny + 2 * H, nx + 2 * H)

    def at(self, a, di=0, dj=0, dk=0, ei=0, ej=0, ek=0):
        """The interior of `a` shifted by (di, dj, dk), with ei, ej, ek more points below."""
        return a[H - ek + dk:H + self.nz + dk, H - ej + dj:H + self.ny + dj, H - ei + di:H + self.nx + di]

    def zeros(self):
        return torch.zeros(self.shape, dtype=F64, device=DEV)

    def periodic(self, a):
        i = H + (torch.arange(self.nx + 2 * H, device=DEV) - H) % self.nx
        j = H + (torch.arange(self.ny + 2 * H, device=DEV) - H) % self.ny
        return a[..., j, :][..., i]

    def reflect(self, a, sign=1.0, staggered=False):
        """The wall conditions in z over a field that is periodic in x and y."""
        a = self.periodic(a)
        k1 = H + self.nz - 1
        if staggered:
            a[H - 1] = 0.0
            a[k1] = 0.0
            for k in range(1, H + 1):
                if k > 1:
                    a[H - k] = sign * a[H + k - 2]
                a[k1 + k] = sign * a[k1 - k]
            return a
        for k in range(1, H + 1):
            a[H - k] = sign * a[H + k - 1]
            a[k1 + k] = sign * a[k1 - k + 1]
        return a


TERRAIN = {  # model, lx, ly, lz [m], stretching exponent
    "hill": ("Boussinesq", 20e3, 1e3, 20e3, 1.0),
    "hills": ("Boussinesq", 100e3, 100e3, 20e3, 1.0),
    "mountain": ("PseudoIncompressible", 100e3, 100e3, 20e3, 1.5),
    "ridges": ("PseudoIncompressible", 400e3, 400e3, 40e3, 1.0),
}


def _topography(terrain, x, y, lx, ly, r):
    """Height [m] over the cell centres x (nx) and y (ny)."""
    X, Y = x[None, :], y[:, None]

    def near(v, c, length):
        return (v - c + length / 2) % length - length / 2

    if terrain == "hill":
        return 250.0 * (1 + torch.cos(math.pi / 10e3 * X)) * r.uniform(0.8, 1.0) + 0 * Y
    if terrain == "mountain":
        return 1000.0 * r.uniform(0.8, 1.0) * torch.exp(-(X ** 2 + Y ** 2) / 10e3 ** 2)
    h = 0 * X + 0 * Y
    ridges = terrain == "ridges"
    for _ in range(20 if ridges else r.randint(1, 5)):
        dx, dy = near(X, r.uniform(-lx / 2, lx / 2), lx), near(Y, r.uniform(-ly / 2, ly / 2), ly)
        top, wide, th = r.uniform(0, 2000.0 if ridges else 1500.0), r.uniform(5e3, 20e3), r.uniform(0, math.pi)
        if ridges:
            dx, dy = dx * math.cos(th) + dy * math.sin(th), (dy * math.cos(th) - dx * math.sin(th)) / 4
        h = h + top * torch.exp(-(dx ** 2 + dy ** 2) / wide ** 2)
    return h * min(1.0, 2000.0 / float(h.max())) if ridges else h


def _fields(box, terrain, r):
    """Grid.jl:173-338 and Atmosphere.jl:278-323 (with compute_n2!.jl) as configs.py uses them, on the GPU."""
    c = constants()
    model, lx, ly, lz, power = TERRAIN[terrain]
    nx, ny, nz = box.nx, box.ny, box.nz
    x = -lx / 2 + (torch.arange(nx, dtype=F64, device=DEV) + 0.5) * (lx / nx)
    y = -ly / 2 + (torch.arange(ny, dtype=F64, device=DEV) + 0.5) * (ly / ny)
    lref = c["lref"]
    top = lz / lref
    dx, dy, dz = lx / lref / nx, ly / lref / ny, top / nz
    hb = torch.zeros(box.shape[1:], dtype=F64, device=DEV)
    hb[H:H + ny, H:H + nx] = _topography(terrain, x, y, lx, ly, r) / lref
    hb = box.periodic(hb)
    # levels of the w-points and of the cell centres
    level = (np.arange(nz + 2 * H) - H + 1) * dz

    def stretch(v):
        return top * (v / top) ** power

    zt = np.where(level < 0, -stretch(np.abs(level)),
                  np.where(level > top, 2 * top - stretch(np.abs(2 * top - level)), stretch(np.abs(level))))
    zs = np.empty_like(zt)
    zs[1:] = 0.5 * (zt[1:] + zt[:-1])
    zs[0] = zt[0] - 0.5 * (zt[2 * H - 1] - zt[2 * H - 2])
    dzt = np.empty_like(zt)
    dzt[1:] = np.diff(zt)
    dzt[0] = zt[2 * H - 1] - zt[2 * H - 2]
    zs = torch.tensor(zs, device=DEV)[:, None, None]
    dzt = torch.tensor(dzt, device=DEV)[:, None, None]
    hx, hy = torch.zeros_like(hb), torch.zeros_like(hb)
    hx[:, 1:-1] = (hb[:, 2:] - hb[:, :-2]) / (2 * dx)
    hy[1:-1] = (hb[2:] - hb[:-2]) / (2 * dy)
    b = (zs - top) / (top - hb)
    f = dict(dx=dx, dy=dy, dz=dz, model=model, zc=(top - hb) / top * zs + hb)
    f["jac"] = (top - hb) / top * dzt / dz
    f["met13"], f["met23"] = (box.periodic(g * b * dz / dzt) for g in (hx, hy))
    f["met33"] = box.periodic(((top / (top - hb)) ** 2 + b ** 2 * (hx ** 2 + hy ** 2)) * (dz / dzt) ** 2)
    if model == "Boussinesq":
        theta = 300.0 / c["thetaref"]
        n2 = ((1e-2 if terrain == "hill" else r.uniform(0.005, 0.02)) * c["tref"]) ** 2
        f["rhobar"] = torch.ones(box.shape, dtype=F64, device=DEV)
        f["thetabar"], f["pbar"], f["n2"] = theta * f["rhobar"], theta * f["rhobar"], n2 * f["rhobar"]
        return f
    t0, p0 = 250.0 / c["thetaref"], 1e5 / c["pref"]
    f["pbar"] = p0 * torch.exp(-c["sig"] * f["zc"] / c["gamma"] / t0)
    f["thetabar"] = t0 * torch.exp(c["kappa"] * c["sig"] / t0 * f["zc"])
    f["rhobar"] = f["pbar"] / f["thetabar"]
    th, jac, k1 = f["thetabar"], f["jac"], H + nz - 1
    n2 = box.zeros()
    n2[H:k1 + 1] = c["g_ndim"] / th[H:k1 + 1] / jac[H:k1 + 1] * 0.5 * (th[H + 1:k1 + 2] - th[H - 1:k1]) / dz
    n2[:H] = c["g_ndim"] / th[H - 1] / jac[H - 1] * (th[H] - th[H - 1]) / dz
    n2[k1 + 1:] = c["g_ndim"] / th[k1 + 1] / jac[k1 + 1] * (th[k1 + 1] - th[k1]) / dz
    f["n2"] = n2
    return f


def _rhs(box, f, terrain, gen):
    """The seeded right-hand side, without its component along the operator's left null vector J fcscal."""
    b = torch.randn((box.nz, box.ny, box.nx), generator=gen, dtype=F64, device=DEV)
    if terrain == "ridges":  # a wave packet plus noise
        lref = constants()["lref"]
        _, lx, ly, lz, _ = TERRAIN[terrain]
        X = ((torch.arange(box.nx, dtype=F64, device=DEV) + 0.5) / box.nx - 0.5)[None, None, :] * lx
        Y = ((torch.arange(box.ny, dtype=F64, device=DEV) + 0.5) / box.ny - 0.5)[None, :, None] * ly
        z = box.at(f["zc"]) * lref
        k = 2 * math.pi / 10e3
        env = torch.exp(-((X / 40e3) ** 2 + (Y / 40e3) ** 2 + ((z - lz / 2) / (lz / 6)) ** 2))
        b = 1e-3 * env * torch.cos(k * X + k * z) + 1e-2 * b
    w = box.at(f["jac"]) * _fcscal(box, f)
    return b - (w * b).sum() / (w * w).sum() * w


def _fcscal(box, f):
    return torch.sqrt(box.at(f["pbar"]) ** 2 / box.at(f["rhobar"]))


def _solve_inputs(case, seed):
    box = Box(case["nx"], case["ny"], case["nz"])
    terrain, r = case["terrain"], random.Random(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    f = _fields(box, terrain, r)
    dt, rf, betar = 1.0, 1.0, box.zeros()
    if terrain == "hill":  # 1 s steps under a sin^2 sponge, rayleigh_factor 1 or 2 as in the time loop
        c = constants()
        dt, rf = 1.0 / c["tref"], float(1 + seed % 2)
        z = f["zc"] * c["lref"]
        betar = torch.where(z >= 10e3, torch.sin(math.pi / 2 * (z - 10e3) / 10e3) ** 2, 0.0) / dt
        betar[:H], betar[H + box.nz:] = betar[H], betar[H + box.nz - 1]
    return box, f, dict(dt=dt, rf=rf, damp=False, rho=box.zeros(), betar=betar), _rhs(box, f, terrain, gen)


def _step_inputs(case, seed):
    """The predictands of the implicit half step; the predictor alone runs the Compressible model, damped, with wave
    tendencies."""
    box, f, st, _ = _solve_inputs(case, seed)
    gen = torch.Generator(device=DEV).manual_seed(seed + 1)

    def noise(a=1.0):
        return a * box.periodic(torch.randn(box.shape, generator=gen, dtype=F64, device=DEV))

    s = dict(u=noise(), v=noise(), w=noise(), rhop=noise(1e-3) * f["rhobar"], pip=noise(), rho=st["rho"])
    if case["kind"] == "predictor":
        f["model"] = "Compressible"
        st.update(dt=0.5, rf=1.0, damp=True, betar=box.periodic(0.1 * torch.rand(box.shape, generator=gen, dtype=F64, device=DEV)),
                  dudt=noise(1e-2), dvdt=noise(1e-2))
        s["rho"] = noise(0.02) * f["rhobar"]
        s["p"] = f["pbar"] * (1 + noise(0.01))
    return box, f, st, s


def _net_inputs(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    b, x = (torch.randn(shape, generator=gen, dtype=torch.float32, device=DEV) for _ in range(2))
    # training problems of the learned part are smaller than the fields it is applied to
    part = tuple(min(n, m) for n, m in zip(shape, (64, 32, 32)))
    tb, tx = (torch.randn(part, generator=gen, dtype=torch.float32, device=DEV).double().cpu().numpy() for _ in range(2))
    params = []
    for name, dims in NET:
        n = math.prod(dims)
        if len(dims) > 1:
            params.append((2 * torch.rand(n, generator=gen, device=DEV) - 1) * math.sqrt(6.0 / dims[-1]))
        else:
            params.append(0.1 * torch.randn(n, generator=gen, device=DEV))
    return b, tb, tx, torch.cat(params)


def _namelist(case):
    return pcf.PoissonNamelist(tolerance=1e-10, tolerance_is_relative=True, poisson_iterations=4000,
                               precision=case.get("precision", "mixed"), multigrid=case.get("multigrid", True), residual="true")


def _solver(box, f):
    s = pcf.PoissonSolver(Domain(box.nx, box.ny, box.nz), f["model"])
    host = {k: v.cpu().numpy() if isinstance(v, torch.Tensor) else v for k, v in f.items() if k != "zc"}
    s.set_grid(host)
    s.set_background(host)
    return s


# ------------------------------------------------------------------- calls --


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        state = _prepare_solve(case, seed)
    elif kind == "ensemble":
        sizes = _member_sizes(case)
        members = [_prepare_solve(dict(terrain="hills", nx=n, ny=n, nz=n // 2, host=False), 1000 * seed + q)
                   for q, n in enumerate(sizes)]
        state = dict(members=members, ensemble=pcf.Ensemble([m["solver"] for m in members]))
    elif kind == "network":
        b, tb, tx, params = _net_inputs(case, seed)
        net = learned.LearnedNet(max_columns=case["nx"] * case["ny"])
        net.set_params(params.cpu().numpy())
        state = dict(net=net, b=b, out=torch.empty_like(b), tb=tb, tx=tx)
    else:
        box, f, st, s = _step_inputs(case, seed)
        state = dict(solver=_solver(box, f), box=box, st=st, start=s, now={k: v.clone() for k, v in s.items()},
                     wold=box.zeros(), dpip=box.zeros())
    state.update(case=case, namelist=_namelist(case))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()  # the library allocates beside torch's pool
    return state


def _prepare_solve(case, seed):
    box, f, st, rhs = _solve_inputs(case, seed)
    state = dict(solver=_solver(box, f), box=box, st=st)
    if case["host"]:
        state.update(rhs=rhs.cpu().numpy(), rho=st["rho"].cpu().numpy(), betar=st["betar"].cpu().numpy(),
                     dpip=np.zeros(box.shape))
    else:
        state.update(rhs=rhs, rho=st["rho"], betar=st["betar"], dpip=box.zeros())
    return state


def _member_sizes(case):
    sizes = [int(n) for n in case["sizes"].split(",")]
    if case["members"] == 32 and sizes == [64, 96, 128, 192]:
        return configs.c4_sizes()
    r = random.Random(case["members"])
    return [r.choice(sizes) for _ in range(case["members"])]


def _pressure(box, dpip):
    """The pressure is determined up to a constant (periodic sides, solid walls): taken without its mean."""
    p = box.at(dpip)
    return p - p.mean()


def run(state):
    kind = state["case"]["kind"]
    # the library works on streams of its own: what torch still does with these arrays has to be done
    torch.cuda.current_stream().synchronize()
    if kind == "solve":
        st = state["st"]
        args = [state[k] if state["case"]["host"] else state[k].data_ptr() for k in ("rhs", "rho", "betar", "dpip")]
        call = state["solver"].solve_poisson if state["case"]["host"] else state["solver"].solve_poisson_device
        info = call(*args[:3], st["dt"], st["rf"], 1.0, state["namelist"], args[3])
        return dict(pressure=_pressure(state["box"], state["dpip"]), converged=not info.errflag)
    if kind == "ensemble":
        ms = state["members"]
        ptr = {k: [m[k].data_ptr() for m in ms] for k in ("rhs", "rho", "betar", "dpip")}
        infos = state["ensemble"].solve_poisson_device(ptr["rhs"], ptr["rho"], ptr["betar"], [m["st"]["dt"] for m in ms],
                                                       [m["st"]["rf"] for m in ms], [1.0] * len(ms), state["namelist"],
                                                       ptr["dpip"])
        return dict(pressure=[_pressure(m["box"], m["dpip"]) for m in ms], converged=all(not i.errflag for i in infos))
    if kind == "network":
        net = state["net"]
        # both on the network's own stream, which gradients() waits for
        net.apply_device(state["b"].data_ptr(), state["out"].data_ptr(), state["b"].shape)
        loss, grads = net.gradients(state["tb"], state["tx"])
        return dict(out=state["out"], loss=loss, grads=grads)
    # the time loop keeps the state before the step (save_backups!) and works on a copy
    now, st = state["now"], state["st"]
    for k, v in state["start"].items():
        now[k].copy_(v)
    torch.cuda.current_stream().synchronize()
    ptr = {k: v.data_ptr() for k, v in now.items()}
    if kind == "predictor":
        state["solver"].implicit_predictor_device(
            st["dt"], st["rf"], ptr["u"], ptr["v"], ptr["w"], ptr["rho"], ptr["rhop"], ptr["pip"], st["betar"].data_ptr(),
            d_p=ptr["p"], d_dudt=st["dudt"].data_ptr(), d_dvdt=st["dvdt"].data_ptr(), d_wold=state["wold"].data_ptr(),
            damp_horizontal_wind_on_rhs=True)
        return dict(now)
    info = state["solver"].implicit_step_device(
        st["dt"], st["rf"], state["namelist"], ptr["u"], ptr["v"], ptr["w"], ptr["rho"], ptr["rhop"], ptr["pip"],
        st["betar"].data_ptr(), state["dpip"].data_ptr(), d_wold=state["wold"].data_ptr())
    out = {k: now[k] for k in ("u", "v", "w", "rho", "rhop")}
    return dict(out, pressure=_pressure(state["box"], state["dpip"]), converged=not info.errflag)


def _cells(case):
    if case["kind"] == "ensemble":
        return sum(n * n * (n // 2) for n in _member_sizes(case))
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Each input read once, each output written once; the operations of one evaluation of what is solved for."""
    n, kind = _cells(case), case["kind"]
    if kind == "network":
        c, t = case["nx"] * case["ny"], min(case["nx"], 32) * min(case["ny"], 32)
        return dict(bytes=8 * n + 16 * t * min(case["nz"], 64) + 8 * NET_SIZE, flops=2 * 172_032 * (c + 3 * t))
    if kind == "predictor":  # 8 grid and background fields, 10 of the state in, 6 out, the backup of w
        return dict(bytes=8 * 25 * n, flops=300 * n)
    if kind == "step":  # the solve's fields and the predictands in and out
        return dict(bytes=8 * (8 + 7 + 7 + 1) * n, flops=600 * n)
    return dict(bytes=8 * (7 + 3 + 1) * n, flops=250 * n)


def tolerance(case):
    if case["kind"] == "network":  # BF16 operands: 6e-3 measured against FP64
        return dict(rel=2.5e-2, max=0.5)
    if case["kind"] == "predictor":  # FP64, pointwise: 5e-16 measured
        return dict(rel=1e-12, max=1e-9)
    # a solve stops at a residual of 1e-10; what is left of it can lie in the smoothest modes, which make up the solution
    # (1e-10 times the square root of the cell count at most).  Measured: 1e-10 to 3e-8, the corrected winds 4e-7.
    return dict(rel=2e-6, max=2e-5)


# ------------------------------------------------------- FP64 in plain torch --

KAPPA = 0.4 / 1.4


def _wind_factors(box, f, s):
    """compute_compressible_wind_factor.jl:102-157 over the haloed grid, at the faces after each cell."""
    if f["model"] != "Compressible":
        one = torch.ones((), dtype=F64, device=DEV)
        return one, one, one
    jp, p, j = f["jac"] * s["p"], s["p"], f["jac"]
    fu, fv, fw = (torch.ones_like(p) for _ in range(3))
    fu[..., :-1] = (jp[..., :-1] + jp[..., 1:]) / 2
    fv[:, :-1] = (jp[:, :-1] + jp[:, 1:]) / 2
    fw[:-1] = j[:-1] * j[1:] * (p[:-1] + p[1:]) / (j[:-1] + j[1:])
    return fu, fv, fw


def _grad_h(box, f, rho, P, d):
    """compute_pressure_gradient.jl for U (d = 0) or V (d = 1), from the face below the first cell on."""
    sh, ext = ((1, 0), dict(ei=1)) if d == 0 else ((0, 1), dict(ej=1))

    def mean(a, dk=0):
        return 0.5 * (box.at(a, 0, 0, dk, **ext) + box.at(a, *sh, dk, **ext))

    dz = mean(P, 1) - mean(P, -1)
    dz[0] = (-mean(P, 2) + 4 * mean(P, 1) - 3 * mean(P))[0]
    dz[-1] = (mean(P, -2) - 4 * mean(P, -1) + 3 * mean(P))[-1]
    diff = (box.at(P, *sh, **ext) - box.at(P, **ext)) / (f["dx"], f["dy"])[d]
    return mean(f["pbar"]) / KAPPA / (mean(rho) + mean(f["rhobar"])) * (
        diff + mean((f["met13"], f["met23"])[d]) * dz * 0.5 / f["dz"])


class Faces:
    """Values at the upper faces of the levels k0 - 1 .. k1: Jacobian-weighted means of a field below and above."""

    def __init__(self, box, f):
        self.box = box
        self.j = self.below(f["jac"])
        self.j1 = self.above(f["jac"])

    def below(self, a, di=0, dj=0):
        return self.box.at(a, di, dj, 0, ek=1)

    def above(self, a, di=0, dj=0):
        return self.box.at(a, di, dj, 1, ek=1)

    def mean(self, a, di=0, dj=0, jac=None):
        j, j1 = (self.j, self.j1) if jac is None else (self.below(jac, di, dj), self.above(jac, di, dj))
        return (j1 * self.below(a, di, dj) + j * self.above(a, di, dj)) / (j + j1)


def _grad_w(box, f, rho, P, z):
    e = {q: z.mean(P, *q, jac=f["jac"]) for q in ((1, 0), (-1, 0), (0, 1), (0, -1))}
    g = z.mean(f["pbar"]) / KAPPA / (z.mean(rho) + z.mean(f["rhobar"])) * (
        z.mean(f["met13"]) * (e[1, 0] - e[-1, 0]) * 0.5 / f["dx"] + z.mean(f["met23"]) * (e[0, 1] - e[0, -1]) * 0.5 / f["dy"]
        + z.mean(f["met33"]) * (z.above(P) - z.below(P)) / f["dz"])
    g[0] = 0.0
    g[-1] = 0.0
    return g


def _buoyancy(box, f, rho, z):
    """compute_buoyancy_factor.jl:108-172 at the upper faces and at the cells."""
    total = rho + f["rhobar"]
    top = f["pbar"] / f["thetabar"] if f["model"] == "Compressible" else f["rhobar"]
    fw = (z.j1 * z.below(top) + z.j * z.above(top)) / (z.j1 * z.below(total) + z.j * z.above(total))
    return fw, box.at(top) / box.at(total)


def _cross(f, z, u, v):
    """met13 u + met23 v, u and v averaged to the cells, below and above each upper face (weighted)."""
    def c(pick):
        return pick(f["met13"]) * (pick(u) + pick(u, -1, 0)) * 0.5 + pick(f["met23"]) * (pick(v) + pick(v, 0, -1)) * 0.5

    return (z.j1 * c(z.below) + z.j * c(z.above)) / (z.j + z.j1)


def _corrections(box, f, st, dpip):
    """What correct!.jl subtracts from u, v, w (haloed arrays) and adds to rhop (interior) for the interior dpip.  Not
    Compressible."""
    P = box.zeros()
    box.at(P)[...] = dpip
    P = box.reflect(P)
    dt, rf, betar, rho, g_ndim = st["dt"], st["rf"], st["betar"], st["rho"], constants()["g_ndim"]
    z = Faces(box, f)
    cu, cv, cw = box.zeros(), box.zeros(), box.zeros()
    box.at(cu, ei=1)[...] = dt * _grad_h(box, f, rho, P, 0)
    box.at(cv, ej=1)[...] = dt * _grad_h(box, f, rho, P, 1)
    fw, fb = _buoyancy(box, f, rho, z)
    n2 = z.mean(f["n2"])
    gw = _grad_w(box, f, rho, P, z)
    inv = 1 / (1 + dt * z.mean(betar) * rf + fw * n2 * dt * dt)
    w = inv * (dt * gw + fw * n2 * dt * dt * _cross(f, z, cu, cv))
    w[0] = 0.0
    w[-1] = 0.0
    box.at(cw, ek=1)[...] = w
    jac, n2c = box.at(f["jac"]), box.at(f["n2"])
    fac = 1 + dt * box.at(betar) * rf
    cross = 0.5 * (box.at(f["met13"]) * (box.at(cu) + box.at(cu, -1)) + box.at(f["met23"]) * (box.at(cv) + box.at(cv, 0, -1)))
    db = -1 / (fac + fb * n2c * dt * dt) * (-fb * n2c * dt * dt * jac * 0.5 * (gw[:-1] + gw[1:])
                                            + fb * n2c * dt * jac * fac * cross)
    return cu, cv, cw, -(box.at(rho) + box.at(f["rhobar"])) / g_ndim * db


def _divergence(box, f, u, v, w):
    """compute_lhs!.jl:68-160 (Boussinesq, PseudoIncompressible)."""
    jp, j, p = f["jac"] * f["pbar"], f["jac"], f["pbar"]
    z = Faces(box, f)
    fu = 0.5 * (box.at(jp, ei=1) + box.at(jp, 1, ei=1)) * box.at(u, ei=1)
    fv = 0.5 * (box.at(jp, ej=1) + box.at(jp, 0, 1, ej=1)) * box.at(v, ej=1)
    fw = z.j * z.j1 * (z.below(p) + z.above(p)) / (z.j + z.j1) * box.at(w, ek=1)
    d = (fu[..., 1:] - fu[..., :-1]) / f["dx"] + (fv[:, 1:] - fv[:, :-1]) / f["dy"] + (fw[1:] - fw[:-1]) / f["dz"]
    return d * KAPPA / box.at(j) / _fcscal(box, f)


def _solve64(box, f, st, rhs):
    """dpip with A dpip = rhs, A q = div(corrections of q), in FP64 to a residual of 1e-13."""
    def apply(q):
        return _divergence(box, f, *_corrections(box, f, st, q)[:3])

    # the operator of the horizontally averaged coefficients, for the preconditioner
    z, dt = Faces(box, f), st["dt"]
    total = st["rho"] + f["rhobar"]
    scale = 1 / _fcscal(box, f)
    c = (dt * box.at(f["pbar"]) ** 2 / box.at(total) * scale).mean((1, 2))
    fw, _ = _buoyancy(box, f, st["rho"], z)
    up = dt / (1 + dt * z.mean(st["betar"]) * st["rf"] + fw * z.mean(f["n2"]) * dt * dt)
    up = up * z.mean(f["pbar"]) / z.mean(total) * z.mean(f["met33"]) * z.j * z.j1 * (z.below(f["pbar"]) + z.above(f["pbar"])) / (z.j + z.j1)
    up[0] = 0.0
    up[-1] = 0.0
    scale = scale / box.at(f["jac"]) / f["dz"] ** 2
    lo, hi = (up[:-1] * scale).mean((1, 2)), (up[1:] * scale).mean((1, 2))
    kx = (2 - 2 * torch.cos(2 * math.pi * torch.arange(box.nx // 2 + 1, dtype=F64, device=DEV) / box.nx)) / f["dx"] ** 2
    ky = (2 - 2 * torch.cos(2 * math.pi * torch.arange(box.ny, dtype=F64, device=DEV) / box.ny)) / f["dy"] ** 2
    k2 = (kx[None, :] + ky[:, None])
    diag = [-c[k] * k2 - lo[k] - hi[k] for k in range(box.nz)]
    ratio, pivot = [], []
    for k in range(box.nz):
        m = diag[k] - (lo[k] * ratio[-1] if k else 0)
        pivot.append(torch.where(m.abs() > 1e-10 * (diag[k].abs() + lo[k] + hi[k]), 1 / m, torch.zeros_like(m)))
        ratio.append(hi[k] * pivot[-1])

    def averaged(r):
        R = torch.fft.rfft2(r)
        for k in range(box.nz):
            R[k] = (R[k] - lo[k] * R[k - 1] if k else R[k]) * pivot[k]
        for k in range(box.nz - 2, -1, -1):
            R[k] -= ratio[k] * R[k + 1]
        return torch.fft.irfft2(R, s=(box.ny, box.nx))

    x, r = torch.zeros_like(rhs), rhs.clone()
    r0, p, first = r.clone(), r.clone(), float(rhs.norm())
    rho = (r * r0).sum()
    for _ in range(80):
        q = averaged(p)
        v = apply(q)
        alpha = rho / (v * r0).sum()
        s = r - alpha * v
        y = averaged(s)
        t = apply(y)
        omega = (t * s).sum() / (t * t).sum()
        x += alpha * q + omega * y
        r = s - omega * t
        if float(r.norm()) <= 1e-13 * first:
            break
        new = (r * r0).sum()
        p = r + alpha / omega * new / rho * (p - omega * v)
        rho = new
    return x


def _predict(box, f, st, s):
    """implicit_integration!.jl:53-63 (update!.jl:632-1336, the Implicit methods)."""
    s = {k: v.clone() for k, v in s.items()}
    dt, rf, betar, g_ndim = st["dt"], st["rf"], st["betar"], constants()["g_ndim"]
    zero = torch.zeros(box.shape, dtype=F64, device=DEV)
    du, dv = st.get("dudt", zero), st.get("dvdt", zero)
    rho, total, jac = s["rho"], s["rho"] + f["rhobar"], f["jac"]
    wold = s["w"].clone()
    fu, fv, fw = (x.expand(box.shape) for x in _wind_factors(box, f, s))
    for name, d, force, jp in (("u", 0, du, fu), ("v", 1, dv, fv)):
        sh, ext = ((1, 0), dict(ei=1)) if d == 0 else ((0, 1), dict(ej=1))
        def mean(a):
            return 0.5 * (box.at(a, **ext) + box.at(a, *sh, **ext))
        fac = 1 + dt * mean(betar) * rf if st["damp"] else 1.0
        here = box.at(s[name], **ext)
        here[...] = (here + dt * (-_grad_h(box, f, rho, s["pip"], d) + mean(force) / mean(total)) * box.at(jp, **ext)) / fac
    z = Faces(box, f)
    fb_w, fb = _buoyancy(box, f, rho, z)
    grad = _grad_w(box, f, rho, s["pip"], z)
    push = f["met13"] * du + f["met23"] * dv
    push = z.mean(push) / z.mean(total)
    n2 = z.mean(f["n2"])
    bb = -g_ndim * (z.j1 * z.below(s["rhop"]) / z.below(total) / z.j + z.j * z.above(s["rhop"]) / z.above(total) / z.j1) / (z.j + z.j1)
    jw = box.at(fw, ek=1)
    w = (box.at(s["w"], ek=1) + dt * jw * (bb - grad + push) + jw * fb_w * n2 * dt * dt * _cross(f, z, s["u"] / fu, s["v"] / fv)) / (
        1 + dt * z.mean(betar) * rf + fb_w * n2 * dt * dt)
    box.at(s["w"], ek=1)[1:-1] = w[1:-1]
    push[0] = 0.0
    push[-1] = 0.0
    s = _walls(box, f, s)
    fu, fv, fw = (x.expand(box.shape) for x in _wind_factors(box, f, s))
    n2, j, fac = box.at(f["n2"]), box.at(jac), 1 + dt * box.at(betar) * rf
    wv = box.at(wold / fw, ek=1)
    wv = 0.5 * (wv[:-1] + wv[1:])
    uu, vv = s["u"] / fu, s["v"] / fv
    cross = 0.5 * (box.at(f["met13"]) * (box.at(uu) + box.at(uu, -1)) + box.at(f["met23"]) * (box.at(vv) + box.at(vv, 0, -1)))
    b = -g_ndim * box.at(s["rhop"]) / box.at(total)
    acc = 0.5 * ((push - grad)[:-1] + (push - grad)[1:])
    b = (-fb * n2 * dt * j * (wv + dt * acc) + fac * b + fb * n2 * dt * j * fac * cross) / (fac + fb * n2 * dt * dt)
    box.at(s["rhop"])[...] = -b * box.at(total) / g_ndim
    return _walls(box, f, s)


def _walls(box, f, s):
    """set_boundaries!(state, BoundaryPredictands()) (rho only where it is a predictand)."""
    sign = dict(u=1.0, v=1.0, w=-1.0, rhop=-1.0, pip=1.0, rho=-1.0, p=1.0)
    return {k: v if k == "rho" and f["model"] == "Boussinesq" else box.reflect(v, sign[k], k == "w") for k, v in s.items()}


NET = [("C1", (64, 576)), ("c1", (64,)), ("W1", (256, 64)), ("b1", (256,)), ("W2", (256, 256)), ("b2", (256,)),
       ("W3", (64, 256)), ("b3", (64,)), ("C2", (64, 576)), ("c2", (64,))]
NET_SIZE = sum(math.prod(d) for _, d in NET)


def _resample(v, n):
    """Rows of v (levels first) at n levels, linearly between level centres."""
    m = v.shape[0]
    if m == n:
        return v
    pos = ((torch.arange(n, dtype=F64, device=DEV) + 0.5) * m / n - 0.5).clamp(0, m - 1)
    k0 = pos.floor().long()
    w = (pos - k0)[:, None, None]
    return (1 - w) * v[k0] + w * v[(k0 + 1).clamp(max=m - 1)]


def _net64(params, b):
    """The columns y of the network (64 levels) for a field of any height."""
    P, o = {}, 0
    for name, dims in NET:
        n = math.prod(dims)
        P[name] = params[o:o + n].reshape(dims)
        o += n

    def windows(v):  # the 3 x 3 neighbours of each column, periodic, tap-major
        return torch.cat([torch.roll(v, (-dj, -di), (1, 2)) for dj in (-1, 0, 1) for di in (-1, 0, 1)])

    def layer(w, c, v):
        return torch.tensordot(P[w], v, 1) + P[c][:, None, None]

    a = torch.relu(layer("C1", "c1", windows(_resample(b, 64))))
    a = torch.relu(layer("W2", "b2", torch.relu(layer("W1", "b1", a))))
    z = layer("W3", "b3", a)
    return z + layer("C2", "c2", windows(z))


def exact(case, seed):
    kind = case["kind"]
    if kind == "network":
        b, tb, tx, params = _net_inputs(case, seed)
        params = params.double().requires_grad_(True)
        with torch.no_grad():
            out = _resample(_net64(params, b.double()), case["nz"])
        t = _resample(torch.tensor(tx, device=DEV), 64)
        loss = ((_net64(params, torch.tensor(tb, device=DEV)) - t) ** 2).sum() / (t ** 2).sum()
        loss.backward()
        return dict(out=out, loss=float(loss), grads=params.grad)
    if kind == "solve":
        box, f, st, rhs = _solve_inputs(case, seed)
        p = _solve64(box, f, st, rhs)
        return dict(pressure=p - p.mean(), converged=None)
    if kind == "ensemble":
        found = []
        for q, n in enumerate(_member_sizes(case)):
            box, f, st, rhs = _solve_inputs(dict(terrain="hills", nx=n, ny=n, nz=n // 2), 1000 * seed + q)
            p = _solve64(box, f, st, rhs)
            found.append(p - p.mean())
        return dict(pressure=found, converged=None)
    box, f, st, s = _step_inputs(case, seed)
    if kind == "predictor":
        return _predict(box, f, st, s)
    st["rho"] = s["rho"]
    s = _predict(box, f, st, _walls(box, f, s))
    p = _solve64(box, f, st, _divergence(box, f, s["u"], s["v"], s["w"]))
    cu, cv, cw, cr = _corrections(box, f, st, p)
    for k, c in (("u", cu), ("v", cv), ("w", cw)):
        s[k] = s[k] - c
    box.at(s["rhop"])[...] += cr
    s = _walls(box, f, s)
    return dict({k: s[k] for k in ("u", "v", "w", "rho", "rhop")}, pressure=p - p.mean(), converged=None)
