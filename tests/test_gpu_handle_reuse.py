"""GPU: one handle (and one ensemble) used for different calls in turn.

What a handle keeps between calls -- captured iteration graphs, the multigrid
hierarchy, the operator in flux form or as planes -- must not reach the next
call's result.  Every kernel sums in a fixed order, so a call on a used handle
gives the bits of the same call on a new one; the residual is checked with the
coefficient planes as well (apply_operator), which no solve of the flux form
shares with it.
"""
import numpy as np
import pytest

from pincflow_poisson import configs as C
from pincflow_poisson import fields as F

pytestmark = pytest.mark.gpu

KW = dict(tolerance=1e-10, tolerance_is_relative=True, poisson_iterations=4000, precision="mixed", multigrid=True)
VCYCLE = dict(mg_dtau=2.0)  # away from its default: asks for the V-cycle


def _grids():
    """Two problems of one shape and model with other spacings, metrics and backgrounds."""
    a = C.c2(nx=48, ny=40, nz=24)
    b = C.c5(nx=48, ny=40, nz=24, lx=60e3, ly=90e3, ridges=2)
    for key in ("dx", "dy", "dz"):
        assert abs(a["fields"][key] / b["fields"][key] - 1) > 0.1
    return a, b


def _handle(pcf, cfg):
    s = pcf.PoissonSolver(cfg["dom"], cfg["model"])
    s.set_grid(cfg["fields"])
    s.set_background(cfg["fields"])
    return s


def _with_density(pcf, cfg, amplitude):
    """cfg with a density fluctuation and a right-hand side in the range of its operator."""
    k = np.arange(cfg["dom"].halo_shape[0])[:, None, None]
    c = dict(cfg, rho=np.ascontiguousarray(amplitude * cfg["fields"]["rhobar"] * np.cos(k)))
    x = np.random.default_rng(7).standard_normal(cfg["dom"].interior_shape)
    with _handle(pcf, c) as s:
        s.compute_operator(c["rho"], c["betar"], c["dt"], c["rayleigh_factor"], return_coef=False)
        c["rhs"] = s.apply_operator(x)
    return c


def _solve(pcf, s, cfg, **nl):
    dpip = np.zeros(cfg["dom"].halo_shape)
    info = s.solve_poisson(cfg["rhs"], cfg["rho"], cfg["betar"], cfg["dt"], cfg["rayleigh_factor"], 1.0,
                           pcf.PoissonNamelist(**dict(KW, **nl)), dpip)
    return cfg["dom"].interior(dpip).copy(), info


def _residual(s, cfg, x):
    """Relative residual of the pressure x with the coefficient planes."""
    r = cfg["rhs"] - s.apply_operator(x * F.fcscal(cfg["dom"], cfg["fields"]) * cfg["dt"])
    return float(np.sqrt((r ** 2).mean() / (cfg["rhs"] ** 2).mean()))


@pytest.mark.parametrize("more", [dict(), VCYCLE], ids=["spectral", "vcycle"])
def test_solve_after_another_grid(pcf, more):
    a, b = _grids()
    with _handle(pcf, a) as s, _handle(pcf, b) as new:
        _, first = _solve(pcf, s, a, **more)
        assert not first.errflag
        s.set_grid(b["fields"])
        s.set_background(b["fields"])
        got, info = _solve(pcf, s, b, **more)
        want, winfo = _solve(pcf, new, b, **more)
        assert not info.errflag and not winfo.errflag
        assert _residual(s, b, got) <= 1.01e-10, _residual(s, b, got)
        assert info.niter == winfo.niter, (info.niter, winfo.niter)
        assert np.array_equal(got, want)


def test_operator_of_the_last_solve_survives_another_grid(pcf):
    """The operator is the last solve's until the next one is made, also where
    the grid has been replaced since."""
    a, b = _grids()
    v = np.random.default_rng(3).standard_normal(a["dom"].interior_shape)
    with _handle(pcf, a) as s, _handle(pcf, a) as ref:
        _solve(pcf, s, a)
        s.set_grid(b["fields"])
        s.set_background(b["fields"])
        ref.compute_operator(a["rho"], a["betar"], a["dt"], a["rayleigh_factor"], return_coef=False)
        assert np.array_equal(s.apply_operator(v), ref.apply_operator(v))


def _device(cfgs):
    import torch
    out = []
    for cfg in cfgs:
        d = {k: torch.from_numpy(np.ascontiguousarray(cfg[k])).cuda() for k in ("rhs", "rho", "betar")}
        d["dpip"] = torch.zeros(cfg["dom"].halo_shape, dtype=torch.float64, device="cuda")
        out.append(d)
    return out


def _solve_ensemble(pcf, ens, cfgs, **nl):
    dev = _device(cfgs)
    infos = ens.solve_poisson_device([d["rhs"].data_ptr() for d in dev], [d["rho"].data_ptr() for d in dev],
                                     [d["betar"].data_ptr() for d in dev], [c["dt"] for c in cfgs],
                                     [c["rayleigh_factor"] for c in cfgs], [c["tolref"] for c in cfgs],
                                     pcf.PoissonNamelist(**dict(KW, **nl)), [d["dpip"].data_ptr() for d in dev])
    return [c["dom"].interior(d["dpip"].cpu().numpy()).copy() for c, d in zip(cfgs, dev)], infos


@pytest.mark.parametrize("more", [dict(), VCYCLE], ids=["spectral", "vcycle"])
def test_ensemble_after_another_grid(pcf, more):
    a, b = _grids()
    other = C.c2(nx=32, ny=24, nz=16, seed=9)
    with _handle(pcf, other) as s0, _handle(pcf, a) as s1, _handle(pcf, other) as n0, _handle(pcf, b) as n1:
        with pcf.Ensemble([s0, s1]) as used, pcf.Ensemble([n0, n1]) as new:
            _, infos = _solve_ensemble(pcf, used, [other, a], **more)
            assert not any(i.errflag for i in infos)
            s1.set_grid(b["fields"])
            s1.set_background(b["fields"])
            got, infos = _solve_ensemble(pcf, used, [other, b], **more)
            want, winfos = _solve_ensemble(pcf, new, [other, b], **more)
        assert not any(i.errflag for i in infos)
        assert _residual(s1, b, got[1]) <= 1.01e-10, _residual(s1, b, got[1])
        assert [i.niter for i in infos] == [i.niter for i in winfos]
        for g, w in zip(got, want):
            assert np.array_equal(g, w)


@pytest.mark.parametrize("first,second", [(dict(), dict(mg_fused_coarse=False)), (dict(mg_operator_bf16=False), dict()),
                                          (dict(mg_smoother_fp8=True), dict()), (dict(mg_min_columns=64), dict())],
                         ids=["fused", "bf16", "fp8", "levels"])
def test_ensemble_after_other_vcycle_settings(pcf, first, second):
    """One ensemble, its V-cycle with one setting after another: each solve
    runs the V-cycle that it asks for (as on new handles)."""
    cfgs = [C.c3(1, nx=32, ny=24, nz=16), C.c3(9, nx=160, ny=16, nz=20)]
    used = [_handle(pcf, c) for c in cfgs]
    try:
        with pcf.Ensemble(used) as ens:
            for more in (first, second, first):
                got, infos = _solve_ensemble(pcf, ens, cfgs, **VCYCLE, **more)
                new = [_handle(pcf, c) for c in cfgs]
                with pcf.Ensemble(new) as fresh:
                    want, winfos = _solve_ensemble(pcf, fresh, cfgs, **VCYCLE, **more)
                for s in new:
                    s.close()
                assert not any(i.errflag for i in infos)
                assert [i.niter for i in infos] == [i.niter for i in winfos]
                for g, w in zip(got, want):
                    assert np.array_equal(g, w)
    finally:
        for s in used:
            s.close()


def test_ensemble_after_a_members_own_solve(pcf):
    """A member that solves by itself with another hierarchy in between has
    freed the level buffers that the ensemble's graph was recorded with."""
    cfgs = [C.c3(1, nx=32, ny=24, nz=16), C.c3(2, nx=48, ny=32, nz=16)]
    used = [_handle(pcf, c) for c in cfgs]
    try:
        with pcf.Ensemble(used) as ens:
            want, winfos = _solve_ensemble(pcf, ens, cfgs, **VCYCLE)
            assert not _solve(pcf, used[1], cfgs[1], mg_min_columns=100)[1].errflag
            got, infos = _solve_ensemble(pcf, ens, cfgs, **VCYCLE)
        assert not any(i.errflag for i in infos) and [i.niter for i in infos] == [i.niter for i in winfos]
        for g, w in zip(got, want):
            assert np.array_equal(g, w)
    finally:
        for s in used:
            s.close()


def test_multigrid_operator_after_a_solve(pcf):
    """pcf_multigrid_operator after a multigrid solve: the hierarchy of that
    solve's operator, whichever preconditioner the solve ran."""
    cfg = C.c2(nx=48, ny=40, nz=24)
    nl = pcf.PoissonNamelist(**KW)
    with _handle(pcf, cfg) as s, _handle(pcf, cfg) as ref:
        for c in (cfg, _with_density(pcf, cfg, 0.1)):  # a second operator on the same handle
            assert not _solve(pcf, s, c)[1].errflag
            ref.compute_operator(c["rho"], c["betar"], c["dt"], c["rayleigh_factor"], return_coef=False)
            levels = ref.multigrid_levels(nl)
            for lv in (1, len(levels) - 1, 0):
                got, want = s.multigrid_operator(lv, levels[lv]), ref.multigrid_operator(lv, levels[lv])
                assert np.array_equal(got, want), lv


def test_no_iterations_allowed(pcf):
    cfg = C.c2(nx=48, ny=40, nz=24)
    with _handle(pcf, cfg) as s:
        for more in (dict(), VCYCLE):
            x, info = _solve(pcf, s, cfg, poisson_iterations=0, **more)
            assert info.errflag and info.niter == 0 and not x.any(), (more, info)


def test_methods_in_turn_on_one_handle(pcf):
    """Spectral, V-cycle and FP64 solves in turn, each with another density,
    give what they give on a new handle."""
    cfg = C.c2(nx=48, ny=40, nz=24)
    with _handle(pcf, cfg) as s:
        for q, more in enumerate([dict(), VCYCLE, dict(), dict(precision="fp64", multigrid=False), dict(), VCYCLE]):
            c = _with_density(pcf, cfg, 0.02 * (q + 1))
            got, info = _solve(pcf, s, c, **more)
            with _handle(pcf, cfg) as new:
                want, winfo = _solve(pcf, new, c, **more)
            assert not info.errflag and info.niter == winfo.niter, (q, info, winfo)
            assert np.array_equal(got, want), q
            if q % 2:  # the component entry point on the operator that the solve left
                x, binfo = s.apply_bicgstab(c["rhs"], 1.0, pcf.PoissonNamelist(**dict(KW, multigrid=False)))
                r = c["rhs"] - s.apply_operator(x)
                assert not binfo.errflag and np.sqrt((r ** 2).mean() / (c["rhs"] ** 2).mean()) <= 1.01e-10
