"""GPU: the column solves and the smallest grids' solver at the edges of their splits.

Column sweeps: 2 to 32 threads per column in runs of at most 8 levels, one
thread per column for up to 8 levels and beyond 128 (FP64) or 256 (FP32); 336
columns are ten and a half warps.  The smallest grids (at most 2048 cells): a
cluster of 8 CTAs that share the columns, one, two or eight cells a thread, with
fewer columns than CTAs, a last CTA with fewer columns, and every cell of 2048.
Tolerances as in the parity suite (test_gpu_parity.py).
"""
import numpy as np
import pytest

from _cases import iterations_agree, oracle_operator, rel_err
from pincflow_poisson import configs as C
from pincflow_poisson import fields as F

pytestmark = pytest.mark.gpu


def _cfg(nx, ny, nz):
    return dict(C.c3(21, nx=nx, ny=ny, nz=nz), damp=False, p=None)


def _drop_null(cfg, x):
    nv = F.fcscal(cfg["dom"], cfg["fields"])
    return x - np.vdot(nv, x) / np.vdot(nv, nv) * nv


def _handle(pcf, cfg):
    s = pcf.PoissonSolver(cfg["dom"], cfg["model"])
    s.set_grid(cfg["fields"])
    s.set_background(cfg["fields"])
    return s


@pytest.mark.parametrize("nz", [8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 256, 257])
def test_column_sweeps(nz, oracle, pcf):
    cfg = _cfg(24, 14, nz)
    d, coef = oracle_operator(oracle, cfg)
    f = cfg["fields"]
    x = np.random.default_rng(6).standard_normal(cfg["dom"].interior_shape)
    with _handle(pcf, cfg) as s:
        s.set_operator(coef)
        for iters in (1, 2):
            ref = oracle.apply_preconditioner(d, coef, f["dx"], f["dy"], 0.8, iters, x)
            nl = pcf.PoissonNamelist(preconditioner_iterations=iters, dtau=0.8)
            assert rel_err(s.apply_preconditioner(x, nl, precision="fp64"), ref) < 1e-12
            assert rel_err(s.apply_preconditioner(x, nl, precision="fp32"), ref) < 1e-4
        # the sweeps that form the iteration's p and s on the way in
        kw = dict(tolerance=1e-10, tolerance_is_relative=True, poisson_iterations=2000)
        ref, rinfo = oracle.bicgstab(d, coef, f["dx"], f["dy"], cfg["rhs"], **kw)
        for precision in ("fp64", "mixed"):
            got, info = s.apply_bicgstab(cfg["rhs"], 1.0, pcf.PoissonNamelist(precision=precision, **kw))
            assert not info.errflag and info.true_residual <= 2e-10, (precision, info)
            assert precision == "mixed" or iterations_agree(info.niter, rinfo["niter"]), (info.niter, rinfo["niter"])
            assert rel_err(_drop_null(cfg, got), _drop_null(cfg, ref)) < 1e-6


@pytest.mark.parametrize("shape", [(16, 16, 8), (5, 7, 58), (3, 3, 200), (20, 3, 33), (4, 2, 256), (4, 1, 512), (3, 1, 600),
                                   (1, 1, 700), (1, 40, 51), (128, 4, 4)], ids=lambda v: "x".join(map(str, v)))
def test_smallest_grids(shape, oracle, pcf):
    cfg = _cfg(*shape)
    d, coef = oracle_operator(oracle, cfg)
    f = cfg["fields"]
    with _handle(pcf, cfg) as s:
        s.set_operator(coef)
        for more in (dict(), dict(preconditioner_iterations=1), dict(preconditioner_iterations=3)):
            kw = dict(tolerance=1e-10, tolerance_is_relative=True, poisson_iterations=2000, **more)
            ref, rinfo = oracle.bicgstab(d, coef, f["dx"], f["dy"], cfg["rhs"], **kw)
            got, info = s.apply_bicgstab(cfg["rhs"], 1.0, pcf.PoissonNamelist(**kw))
            assert not rinfo["errflag"] and not info.errflag, (more, info, rinfo)
            assert iterations_agree(info.niter, rinfo["niter"]), (more, info.niter, rinfo["niter"])
            assert rel_err(_drop_null(cfg, got), _drop_null(cfg, ref)) < 1e-6, more
        # without the preconditioner: a few iterations, step by step as the oracle's
        kw = dict(tolerance=1e-30, tolerance_is_relative=True, poisson_iterations=4, preconditioner=False)
        ref, rinfo = oracle.bicgstab(d, coef, f["dx"], f["dy"], cfg["rhs"], **kw)
        got, info = s.apply_bicgstab(cfg["rhs"], 1.0, pcf.PoissonNamelist(**kw))
        assert info.errflag and info.niter == 4 and rel_err(got, ref) < 1e-9
