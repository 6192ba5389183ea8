"""GPU: batched solves of uneven ensemble members (pcf_ensemble_*) against
each member's own single-handle solve and the CPU oracle.

The ensemble runs the same device-side iteration as a single handle, so each
member's iteration count must equal its single-handle count and its pressure
agree to 1e-12 (relative to its largest magnitude); against the oracle's
plain FP64 solve the pressure agrees to 1e-6 (null space removed).  Members
run the spectral preconditioner by default and the V-cycle where a setting
asks for it."""
import numpy as np
import pytest

from _cases import rel_err

pytestmark = pytest.mark.gpu

SIZES = [32, 48, 64, 32, 40]
NL = dict(tolerance=1e-10, tolerance_is_relative=True, poisson_iterations=4000, precision="mixed",
          multigrid=True, residual="true")


@pytest.fixture(scope="module")
def members(pcf):
    import torch
    from pincflow_poisson import configs as C
    out = []
    for q, nx in enumerate(SIZES):
        cfg = C.c4(q, nx)
        if q == 3:
            cfg["rhs"] = np.zeros_like(cfg["rhs"])  # a member with nothing to solve
        s = pcf.PoissonSolver(cfg["dom"], cfg["model"])
        s.set_grid(cfg["fields"])
        s.set_background(cfg["fields"])
        dev = {k: torch.from_numpy(np.ascontiguousarray(cfg[k])).cuda() for k in ("rhs", "rho", "betar")}
        dev["dpip"] = torch.zeros(cfg["dom"].halo_shape, dtype=torch.float64, device="cuda")
        out.append((cfg, s, dev))
    yield out
    for _, s, _ in out:
        s.close()


def _solve_ensemble(pcf, ens, members, nl):
    return ens.solve_poisson_device([d["rhs"].data_ptr() for _, _, d in members],
                                    [d["rho"].data_ptr() for _, _, d in members],
                                    [d["betar"].data_ptr() for _, _, d in members],
                                    [c["dt"] for c, _, _ in members], [c["rayleigh_factor"] for c, _, _ in members],
                                    [c["tolref"] for c, _, _ in members], nl,
                                    [d["dpip"].data_ptr() for _, _, d in members])


# mg_dtau away from its default asks for the V-cycle in place of the spectral preconditioner
@pytest.mark.parametrize("more", [dict(), dict(mg_dtau=2.0)], ids=["spectral", "vcycle"])
@pytest.mark.parametrize("fused", [None, False])
def test_ensemble_matches_single_solves(pcf, members, fused, more):
    """fused None: the default, the V-cycle's coarse levels as one cluster
    launch in the ensemble; False: one kernel per step as in single solves
    (the spectral preconditioner has no coarse levels: no difference there)."""
    nl = pcf.PoissonNamelist(**NL, mg_fused_coarse=fused, **more)
    with pcf.Ensemble([s for _, s, _ in members]) as ens:
        infos = _solve_ensemble(pcf, ens, members, nl)
        got = [d["dpip"].cpu().numpy().copy() for _, _, d in members]
        # the same graph serves a second call
        infos2 = _solve_ensemble(pcf, ens, members, nl)
        again = [d["dpip"].cpu().numpy().copy() for _, _, d in members]
        assert ens.launch_count > 0
    for q, (cfg, s, d) in enumerate(members):
        info = infos[q]
        assert not info.errflag, (q, info)
        assert infos2[q].niter == info.niter
        assert rel_err(again[q], got[q]) <= 1e-12 if np.abs(got[q]).max() > 0 else np.abs(again[q]).max() == 0
        if q == 3:
            assert info.niter == 0 and np.abs(got[q]).max() == 0
            continue
        assert info.true_residual <= 1e-10
        d["dpip"].zero_()
        # the ensemble runs the V-cycle's coarse levels as one cluster launch by
        # default (mg_fused_coarse = -1); the single solve is asked for the same
        single = s.solve_poisson_device(d["rhs"].data_ptr(), d["rho"].data_ptr(), d["betar"].data_ptr(), cfg["dt"],
                                        cfg["rayleigh_factor"], cfg["tolref"],
                                        pcf.PoissonNamelist(**NL, mg_fused_coarse=fused is None, **more),
                                        d["dpip"].data_ptr())
        ref = d["dpip"].cpu().numpy()
        assert single.niter == info.niter, (q, single.niter, info.niter)
        assert rel_err(got[q], ref) <= 1e-12, (q, rel_err(got[q], ref))


def test_ensemble_pressure_matches_oracle(pcf, oracle, members):
    from _cases import oracle_operator
    cfg, s, d = members[1]
    nl = pcf.PoissonNamelist(**NL)
    with pcf.Ensemble([m[1] for m in members]) as ens:
        infos = _solve_ensemble(pcf, ens, members, nl)
    assert not infos[1].errflag
    cfg = dict(cfg, damp=False, p=None)
    od, coef = oracle_operator(oracle, cfg)
    f = cfg["fields"]
    ref = oracle.solve_poisson(od, oracle.MODELS[cfg["model"]], f, cfg["rho"], cfg["betar"], cfg["rhs"], cfg["dt"],
                               cfg["rayleigh_factor"], tolerance=1e-12, tolerance_is_relative=True,
                               poisson_iterations=4000)[0]
    dom = cfg["dom"]
    a, b = dom.interior(d["dpip"].cpu().numpy()), dom.interior(ref)
    assert rel_err(a - a.mean(), b - b.mean()) < 1e-6


@pytest.mark.parametrize("more", [dict(), dict(mg_dtau=2.0)], ids=["spectral", "vcycle"])
def test_ensemble_with_autotuner(pcf, members, more):
    """The stencils are tuned in either case; the V-cycle solve launches them
    (the spectral one only where it falls back to the V-cycle)."""
    pcf.autotune_clear()
    nl = pcf.PoissonNamelist(**NL, autotune=True, **more)
    with pcf.Ensemble([s for _, s, _ in members]) as ens:
        infos = _solve_ensemble(pcf, ens, members, nl)
    assert all(not i.errflag for i in infos)
    entries = pcf.autotune_entries()
    sizes = {(e["nx"], e["ny"], e["nz"]) for e in entries if e["kernel"] == "total32_diff"}
    assert sizes == {(nx, nx, nx // 2) for nx in set(SIZES)}
    for e in entries:
        assert e["tile_x"] in (32, 16, 8) and 2 <= e["levels"] <= e["nz"]
        if e["ms_default"] > 0:  # the heuristic shape is one of the candidates
            assert e["ms_best"] <= e["ms_default"]
    pcf.autotune_clear()


def test_ensemble_rejects_what_it_does_not_run(pcf, members):
    solvers = [s for _, s, _ in members]
    with pytest.raises(pcf.PoissonError):
        pcf.Ensemble([solvers[0], solvers[0]])
    with pcf.Ensemble(solvers) as ens:
        with pytest.raises(pcf.PoissonError) as e:
            _solve_ensemble(pcf, ens, members, pcf.PoissonNamelist(**dict(NL, precision="fp64", multigrid=False)))
        assert e.value.code == pcf._lib.PCF_EINVAL


def _ensemble_of(pcf, cfgs, solvers, **nl):
    """(pressures, infos) of one ensemble solve of cfgs on the given solvers."""
    import torch
    members = []
    for cfg, s in zip(cfgs, solvers):
        dev = {k: torch.from_numpy(np.ascontiguousarray(cfg[k])).cuda() for k in ("rhs", "rho", "betar")}
        dev["dpip"] = torch.zeros(cfg["dom"].halo_shape, dtype=torch.float64, device="cuda")
        members.append((cfg, s, dev))

    def solve(ens):
        infos = _solve_ensemble(pcf, ens, members, pcf.PoissonNamelist(**dict(NL, **nl)))
        return [c["dom"].interior(d["dpip"].cpu().numpy()).copy() for c, _, d in members], infos
    return solve


def _solvers(pcf, cfgs):
    out = []
    for cfg in cfgs:
        s = pcf.PoissonSolver(cfg["dom"], cfg["model"])
        s.set_grid(cfg["fields"])
        s.set_background(cfg["fields"])
        out.append(s)
    return out


def _residual(s, cfg, x):
    """Relative residual of the pressure x with the member's coefficient planes."""
    from pincflow_poisson import fields as F
    r = cfg["rhs"] - s.apply_operator(x * F.fcscal(cfg["dom"], cfg["fields"]) * cfg["dt"])
    return float(np.sqrt((r ** 2).mean() / (cfg["rhs"] ** 2).mean()))


def test_ensemble_with_uneven_halos(pcf):
    """Halo columns that are not the periodic image of the interior (the flux
    form cannot tell them apart, the coefficient planes can): a member that
    has them in the second of three solves."""
    from pincflow_poisson import configs as C
    a, b = C.c2(nx=32, ny=24, nz=16, seed=9), C.c2(nx=32, ny=16, nz=12, seed=3)
    rng = np.random.default_rng(11)
    u = dict(b, rho=0.05 * rng.standard_normal(b["dom"].halo_shape) * b["fields"]["rhobar"])
    used = _solvers(pcf, [a, b])
    used[1].compute_operator(u["rho"], u["betar"], u["dt"], u["rayleigh_factor"], return_coef=False)
    u["rhs"] = used[1].apply_operator(rng.standard_normal(b["dom"].interior_shape))
    try:
        with pcf.Ensemble(used) as ens:
            for cfgs in ([a, b], [a, u], [a, b]):
                got, infos = _ensemble_of(pcf, cfgs, used)(ens)
                new = _solvers(pcf, cfgs)
                with pcf.Ensemble(new) as fresh:
                    want, winfos = _ensemble_of(pcf, cfgs, new)(fresh)
                for s in new:
                    s.close()
                assert [i.niter for i in infos] == [i.niter for i in winfos]
                for q, cfg in enumerate(cfgs):
                    assert not infos[q].errflag and infos[q].niter <= 12, (q, infos[q])
                    assert np.array_equal(got[q], want[q])
                    assert _residual(used[q], cfg, got[q]) <= 1.01e-10
    finally:
        for s in used:
            s.close()


def test_ensemble_member_falls_back_to_the_vcycle(pcf):
    """One member whose background density varies by e^8 along x, about which
    the horizontal averages say nothing: it goes on with the V-cycle after the
    24 spectral iterations, the other member is unaffected."""
    from pincflow_poisson import configs as C
    from pincflow_poisson import fields as F
    a, b = C.c2(nx=32, ny=24, nz=16, seed=9), C.c2(nx=64, ny=32, nz=16)
    f = dict(b["fields"])
    x = 2 * np.pi * (np.arange(b["dom"].nx + 6) - 3) / b["dom"].nx
    f["rhobar"] = f["rhobar"] * np.exp(4 * np.cos(x))[None, None, :]
    b = dict(b, fields=f, rhs=F.consistent_projection(b["dom"], f, b["rhs"]))
    solvers = _solvers(pcf, [a, b])
    try:
        with pcf.Ensemble(solvers) as ens:
            solve = _ensemble_of(pcf, [a, b], solvers, tolerance=1e-8)
            got, infos = solve(ens)
            again, infos2 = solve(ens)
        print("iterations:", [i.niter for i in infos])
        assert infos[0].niter <= 12 < 24 < infos[1].niter
        for q, cfg in enumerate((a, b)):
            assert not infos[q].errflag and infos[q].true_residual <= 1e-8, infos[q]
            assert _residual(solvers[q], cfg, got[q]) <= 1.01e-8
            assert infos2[q].niter == infos[q].niter and np.array_equal(again[q], got[q])
    finally:
        for s in solvers:
            s.close()
