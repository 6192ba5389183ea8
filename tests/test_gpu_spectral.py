"""GPU: the spectral preconditioner of the mixed solve.

pcf_apply_spectral against its definition in FP64 numpy (transform the
right-hand side along x and y, solve the tridiagonal systems of the level
means along z, transform back), on grids that reach every radix of the
transforms (8, 4, 2, 3, 5, 7 and primes by their definition), odd and even
extents, one cell along y, partial blocks of rows and columns, and runs of 4,
8 and 16 levels.  The operator's defect is set away from zero, so that the
constant mode is determined.

Tolerance: the FP32 transforms and pivots round at 2^-24 per operation; a
value passes through at most 2 (log2 nx + log2 ny) + 2 nz of them, whose
errors add up like their square root against the result's norm: 2^-24
sqrt(2 (12 + 12) + 1024) = 2e-6; the constant mode, and modes near it, amplify
the sums' rounding by the ratio of the largest eigenvalue to their own, which
the defect set here bounds by 20: 4e-5 norm-wise.

Solves with the spectral preconditioner: the FP64 true residual, the pressure
of the V-cycle's solve within 1e-6 (the constant removed), in at most 12
iterations on every parity case (rho and comp have halo columns that are not
the periodic image of the interior, so they apply the coefficient planes; the
others apply the operator in flux form).
"""
import numpy as np
import pytest

from _cases import case, consistent_rhs, rel_err
from pincflow_poisson import configs as C
from pincflow_poisson import fields as F

pytestmark = pytest.mark.gpu

# (nx, ny, nz): radices 8.8 / 8.4 | 3.5 / 7 | prime 37, 29 | 2 | one row along y | 16-level runs | 8-level runs
SHAPES = [(64, 32, 16), (60, 42, 13), (37, 29, 12), (14, 22, 5), (40, 1, 40), (8, 6, 300), (512, 10, 192), (1, 96, 8),
          (250, 144, 33)]


def _averaged_inverse(planes, fch, b):
    """The definition in FP64: planes (25, nz, ny, nx) of A, fch haloed."""
    nz, ny, nx = b.shape
    from pincflow_poisson.fields import Domain
    dom = Domain(nx, ny, nz)
    off = {1: (-1, 0, 0), 2: (1, 0, 0), 3: (0, -1, 0), 4: (0, 1, 0), 5: (0, 0, -1), 6: (0, 0, 1)}

    def nb(di, dj, dk):
        return fch[3 + dk:3 + dk + nz, 3 + dj:3 + dj + ny, 3 + di:3 + di + nx]

    mean = {p: (planes[p] * nb(*o)).mean(axis=(1, 2)) for p, o in off.items()}
    d = 0.0
    names = ["", "l", "r", "b", "f", "d", "u", "ld", "lu", "rd", "ru", "bd", "bu", "fd", "fu", "dd", "uu", "ldd", "luu",
             "rdd", "ruu", "bdd", "buu", "fdd", "fuu"]
    for p, s in enumerate(names):
        o = (s.count("r") - s.count("l"), s.count("f") - s.count("b"), s.count("u") - s.count("d"))
        d = d + planes[p] * nb(*o)
    d = d.mean(axis=(1, 2))
    cx, cy, ad, au = (mean[1] + mean[2]) / 2, (mean[3] + mean[4]) / 2, mean[5].copy(), mean[6].copy()
    ad[0] = au[-1] = 0.0
    ex = 2 * np.cos(2 * np.pi * np.arange(nx) / nx) - 2
    ey = 2 * np.cos(2 * np.pi * np.arange(ny) / ny) - 2
    R = np.fft.fft2(b)
    lam = (d - ad - au)[:, None, None] + cx[:, None, None] * ex[None, None, :] + cy[:, None, None] * ey[None, :, None]
    piv, ratio = np.empty_like(lam), np.empty_like(lam)
    for k in range(nz):
        piv[k] = 1 / (lam[k] - (ad[k] * ratio[k - 1] if k else 0))
        ratio[k] = au[k] * piv[k]
        R[k] = (R[k] - (ad[k] * R[k - 1] if k else 0)) * piv[k]
    for k in range(nz - 2, -1, -1):
        R[k] -= ratio[k] * R[k + 1]
    assert dom.interior_shape == R.shape
    return np.fft.ifft2(R).real


@pytest.mark.parametrize("shape", SHAPES)
def test_spectral_inverse_matches_its_definition(shape, pcf):
    nx, ny, nz = shape
    cfg = C.c3(3, nx=nx, ny=ny, nz=nz)
    dom, f = cfg["dom"], cfg["fields"]
    with pcf.PoissonSolver(dom, cfg["model"]) as s:
        s.set_grid(f)
        s.set_background(f)
        planes = s.compute_operator(cfg["rho"], cfg["betar"], cfg["dt"], cfg["rayleigh_factor"])
        planes[0] -= 0.05 * np.abs(planes[0]).max()  # a defect: no free constant
        s.set_operator(planes)
        b = np.random.default_rng(nx + ny).standard_normal(dom.interior_shape)
        got = s.apply_spectral(b)
        again = s.apply_spectral(b)
    want = _averaged_inverse(planes, np.sqrt(f["pbar"] ** 2 / f["rhobar"]), b)
    assert np.array_equal(got, again)
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err <= 4e-5, err


@pytest.mark.parametrize("name", ["mtn", "odd", "rho", "comp", "wide", "oddx", "wide2", "wide3"])
def test_spectral_solve_matches_the_vcycle(name, oracle, pcf):
    cfg = case(name)
    dom = cfg["dom"]
    rhs = consistent_rhs(oracle, cfg)
    kw = dict(tolerance=1e-10, tolerance_is_relative=True, poisson_iterations=4000, precision="mixed", multigrid=True,
              damp_horizontal_wind_on_rhs=cfg["damp"])
    out = []
    with pcf.PoissonSolver(dom, cfg["model"]) as s:
        s.set_grid(cfg["fields"])
        s.set_background(cfg["fields"])
        for more in (dict(), dict(mg_dtau=2.0)):  # mg_dtau away from its default asks for the V-cycle
            dpip = np.zeros(dom.halo_shape)
            info = s.solve_poisson(rhs, cfg["rho"], cfg["betar"], cfg["dt"], cfg["rayleigh_factor"], 1.0,
                                   pcf.PoissonNamelist(**kw, **more), dpip, p=cfg["p"])
            assert not info.errflag and info.true_residual <= 1e-10, info
            out.append((dom.interior(dpip).copy(), info.niter))
            # the residual with the coefficient planes (assembled on demand after a
            # spectral solve), independent of the form the solve applied
            x = dom.interior(dpip) * F.fcscal(dom, cfg["fields"]) * cfg["dt"]
            r = rhs - s.apply_operator(x)
            assert np.sqrt((r ** 2).mean() / (rhs ** 2).mean()) <= 1.01e-10
    (a, na), (b, nb) = out
    assert na <= 12 and na < nb, (na, nb)
    assert rel_err(a - a.mean(), b - b.mean()) < 1e-6


def test_spectral_solve_falls_back_to_the_vcycle(pcf):
    """A horizontally averaged operator says nothing about this one: the
    background density varies by e^8 along x, so the spectral iteration does
    not converge in its 24 iterations and the solve goes on with the V-cycle,
    within the V-cycle's own count plus those."""
    cfg = C.c2(nx=64, ny=32, nz=16)
    dom, f = cfg["dom"], dict(cfg["fields"])
    x = 2 * np.pi * (np.arange(dom.nx + 6) - 3) / dom.nx
    f["rhobar"] = f["rhobar"] * np.exp(4 * np.cos(x))[None, None, :]
    rhs = F.consistent_projection(dom, f, cfg["rhs"])
    kw = dict(tolerance=1e-8, tolerance_is_relative=True, poisson_iterations=4000, precision="mixed", multigrid=True)
    counts = []
    with pcf.PoissonSolver(dom, cfg["model"]) as s:
        s.set_grid(f)
        s.set_background(f)
        for more in (dict(), dict(mg_dtau=2.4)):
            dpip = np.zeros(dom.halo_shape)
            info = s.solve_poisson(rhs, cfg["rho"], cfg["betar"], cfg["dt"], cfg["rayleigh_factor"], 1.0,
                                   pcf.PoissonNamelist(max_refinements=0, **kw, **more), dpip)
            assert not info.errflag and info.true_residual <= 1e-8, (more, info)
            counts.append(info.niter)
    print("iterations with the fallback / V-cycle alone:", counts)
    # BiCGSTAB counts move by a few iterations with the pseudo-time step and the start
    assert 24 < counts[0] <= 24 + counts[1] + max(8, 0.15 * counts[1]), counts


def _after_a_solve(pcf, cfg):
    """A handle whose operator is held in flux form (a default multigrid solve, one iteration)."""
    s = pcf.PoissonSolver(cfg["dom"], cfg["model"])
    s.set_grid(cfg["fields"])
    s.set_background(cfg["fields"])
    s.solve_poisson(np.ascontiguousarray(cfg["rhs"]), cfg["rho"], cfg["betar"], cfg["dt"], cfg["rayleigh_factor"], 1.0,
                    pcf.PoissonNamelist(precision="mixed", multigrid=True, poisson_iterations=1,
                                        damp_horizontal_wind_on_rhs=cfg.get("damp", False)),
                    np.zeros(cfg["dom"].halo_shape), p=cfg.get("p"))
    return s


def _periodic(dom, a):
    """a with the periodic image of the interior in its halo columns."""
    i = (np.arange(dom.nx + 6) - 3) % dom.nx + 3
    j = (np.arange(dom.ny + 6) - 3) % dom.ny + 3
    return np.ascontiguousarray(a[:, j][:, :, i])


@pytest.mark.parametrize("name", ["mtn", "odd", "rho", "comp", "wide", "wide2"])
def test_flux_form_matches_the_planes(name, pcf):
    """The flux form against the coefficient planes, both from the same fields
    (with even halos).  A coefficient is a product of about 20 factors and a
    sum of a few such products, which cancel in the row's sum: 1e-13 of the
    largest result in FP64, 2^29 times as much, 5e-5, in FP32."""
    cfg = dict(case(name))
    dom = cfg["dom"]
    for key in ("rho", "betar", "p"):
        if cfg[key] is not None:
            cfg[key] = _periodic(dom, cfg[key])
    pi = np.random.default_rng(5).standard_normal(dom.interior_shape)
    with _after_a_solve(pcf, cfg) as s:
        got = s.apply_flux(pi)
        got32 = s.apply_flux(pi, "fp32")
        want = s.apply_operator(pi * F.fcscal(dom, cfg["fields"]))
        with pytest.raises(pcf.PoissonError) as e:  # apply_operator assembled the planes
            s.apply_flux(pi)
        assert e.value.code == pcf._lib.PCF_ENOTREADY
    print(f"{name}: {rel_err(got, want):.1e} {rel_err(got32, want):.1e}")
    assert rel_err(got, want) <= 1e-13 and rel_err(got32, want) <= 5e-5


@pytest.mark.parametrize("name", ["mtn", "odd", "wide", "wide2"])
def test_flux_form_of_a_constant_is_zero(name, pcf):
    """Exactly, in either precision and also where multiples of the constant
    round: every term is a difference of pressures."""
    cfg = case(name)
    with _after_a_solve(pcf, cfg) as s:
        for value in (1.0, 1 / 3, -0.7e5, np.pi):
            pi = np.full(cfg["dom"].interior_shape, value)
            for precision in ("fp64", "fp32"):
                assert not s.apply_flux(pi, precision).any(), (value, precision)


@pytest.mark.parametrize("name", ["rho", "comp", "200x1x40", "1x100x30"])
def test_solve_in_flux_form(name, pcf):
    """Solves that end in the flux form: density, damping and the Compressible
    model with even halos, and grids of one row along x or y."""
    if "x" in name:
        nx, ny, nz = (int(v) for v in name.split("x"))
        cfg = dict(C.c3(31, nx=nx, ny=ny, nz=nz), damp=False, p=None)
    else:
        cfg = dict(case(name))
    dom = cfg["dom"]
    for key in ("rho", "betar", "p"):
        if cfg[key] is not None:
            cfg[key] = _periodic(dom, cfg[key])
    with pcf.PoissonSolver(dom, cfg["model"]) as s:
        s.set_grid(cfg["fields"])
        s.set_background(cfg["fields"])
        s.compute_operator(cfg["rho"], cfg["betar"], cfg["dt"], cfg["rayleigh_factor"], cfg["damp"], cfg["p"],
                           return_coef=False)
        want = np.random.default_rng(9).standard_normal(dom.interior_shape)
        rhs = s.apply_operator(want)
        dpip = np.zeros(dom.halo_shape)
        info = s.solve_poisson(rhs, cfg["rho"], cfg["betar"], cfg["dt"], cfg["rayleigh_factor"], 1.0,
                               pcf.PoissonNamelist(tolerance=1e-10, tolerance_is_relative=True, precision="mixed",
                                                   multigrid=True, damp_horizontal_wind_on_rhs=cfg["damp"]),
                               dpip, p=cfg["p"])
        assert not info.errflag and info.niter <= 12, info
        fc = F.fcscal(dom, cfg["fields"])
        x = dom.interior(dpip) * fc * cfg["dt"]
        s.apply_flux(x / fc)  # (an error if the solve went on with the planes)
        r = rhs - s.apply_operator(x)
        assert np.sqrt((r ** 2).mean() / (rhs ** 2).mean()) <= 1.01e-10
    got, want = x / fc, want / fc
    if cfg["model"] != "Compressible":  # the pressure's free constant
        got, want = got - got.mean(), want - want.mean()
    assert rel_err(got, want) < 1e-6
