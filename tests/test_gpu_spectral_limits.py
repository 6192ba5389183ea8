"""GPU: grids at and beyond the limits of the spectral solve's kernels.

Beyond a limit a default multigrid solve runs the V-cycle: more than 4096 cells
along x or y, more than 512 levels, or more columns than the flux-form apply
has partial sums for (16384 tiles of 32 x 4 columns).  Either way the solve
reaches the FP64 true residual, checked with the coefficient planes.
"""
import numpy as np
import pytest

from pincflow_poisson import configs as C
from pincflow_poisson import fields as F

pytestmark = pytest.mark.gpu

KW = dict(tolerance=1e-9, tolerance_is_relative=True, poisson_iterations=4000, precision="mixed", multigrid=True)


def _problem(nx, ny, nz, cell):
    """The large domain's terrain family with cells of `cell` metres."""
    return C.c5(nx=nx, ny=ny, nz=nz, lx=cell * nx, ly=cell * ny, ridges=3)


# (nx, ny, nz, metres per cell): the longest lines, primes above 37, runs of 16 levels up to the last one, and the
# most columns (2,097,152)
WITHIN = [(4096, 8, 16, 5e3), (8, 4096, 16, 5e3), (127, 41, 16, 1e3), (40, 24, 300, 1e3), (16, 24, 512, 1e3),
          (2048, 1024, 4, 5e3)]
# one more of each; iterations allowed (the V-cycle does not converge on grids 8 cells wide and 4104 long)
BEYOND = [(4104, 8, 16, 5e3, 2), (8, 4104, 16, 5e3, 2), (16, 24, 513, 1e3, 4000), (2112, 1024, 4, 5e3, 4000)]


def _solve(pcf, s, cfg, **nl):
    dpip = np.zeros(cfg["dom"].halo_shape)
    info = s.solve_poisson(cfg["rhs"], cfg["rho"], cfg["betar"], cfg["dt"], cfg["rayleigh_factor"], 1.0,
                           pcf.PoissonNamelist(**dict(KW, **nl)), dpip)
    return dpip, info


def _residual(s, cfg, dpip):
    dom = cfg["dom"]
    r = cfg["rhs"] - s.apply_operator(dom.interior(dpip) * F.fcscal(dom, cfg["fields"]) * cfg["dt"])
    return np.sqrt((r ** 2).mean() / (cfg["rhs"] ** 2).mean())


@pytest.mark.parametrize("nx,ny,nz,cell", WITHIN)
def test_solve_within_the_limits(nx, ny, nz, cell, pcf):
    cfg = _problem(nx, ny, nz, cell)
    with pcf.PoissonSolver(cfg["dom"], cfg["model"]) as s:
        s.set_grid(cfg["fields"])
        s.set_background(cfg["fields"])
        s.profile(True)
        dpip, info = _solve(pcf, s, cfg)
        prof = s.profile_read()
        s.profile(False)
        assert not info.errflag and info.true_residual <= 1e-9 and info.niter <= 12, info
        assert prof["spectral"]["count"] > 0 and prof["thomas32"]["count"] == 0
        graph, again = _solve(pcf, s, cfg)  # as one graph launch (off while profiling)
        assert again.niter == info.niter and np.array_equal(graph, dpip)
        assert _residual(s, cfg, dpip) <= 1.01e-9


@pytest.mark.parametrize("nx,ny,nz,cell,iterations", BEYOND)
def test_solve_beyond_the_limits(nx, ny, nz, cell, iterations, pcf):
    cfg = _problem(nx, ny, nz, cell)
    with pcf.PoissonSolver(cfg["dom"], cfg["model"]) as s:
        s.set_grid(cfg["fields"])
        s.set_background(cfg["fields"])
        s.profile(True)
        dpip, info = _solve(pcf, s, cfg, poisson_iterations=iterations)
        prof = s.profile_read()
        print(f"{nx} x {ny} x {nz}: {info.niter} iterations")
        assert prof["spectral"]["count"] == 0 and prof["thomas32"]["count"] > 0
        if iterations == 2:
            assert info.errflag and info.niter == 2
        else:
            assert not info.errflag and info.true_residual <= 1e-9, info
            assert _residual(s, cfg, dpip) <= 1.01e-9
