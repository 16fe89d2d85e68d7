"""Mixed precision on Jacobians that FP32 factors do not precondition: steady
Newton far from a solution, where the pivot blocks are ill conditioned."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

IMAX, JMAX = 65, 49


def solver(v2d, oracle_mod, precision, re=600.0, **config):
    xg, yg = oracle_mod.generate_cylinder(IMAX, JMAX)
    return v2d.Solver(v2d.Config(verbose=False, write_csv=False, write_xdmf=False,
                                 compute_forces=False, re=re, alpha_deg=5.0, steady=True,
                                 precision=precision, ksp_restart=30, krylov_max_it=60, **config),
                      mesh=(xg, yg))


def far_state(v2d, oracle_mod, steps=5):
    """The state after a few Newton steps from the free stream in FP64."""
    s = solver(v2d, oracle_mod, "fp64")
    for _ in range(steps):
        code, _, lin = s.dev.newton(0.0)
        assert code == 0 and lin.converged
    st = [a.copy() for a in s.dev.get_state()]
    s.set_state(*st)
    assert s.dev.newton(0.0)[0] == 0
    want = np.concatenate(s.dev.get_state()[:2])
    s.close()
    return st, want


@pytest.mark.parametrize("factors", ["fp32", "fp64"])
@pytest.mark.parametrize("reuse", [0, 8])
def test_newton_converges_where_fp32_factors_do_not(v2d, oracle_mod, factors, reuse):
    """The update agrees with FP64's to what the solve's tolerance (1e-10 of the
    residual, both) leaves of it at a condition of up to 1e8 in this norm."""
    st, want = far_state(v2d, oracle_mod)
    s = solver(v2d, oracle_mod, "mixed", lu_factors=factors, lu_reuse_its=reuse)
    for _ in range(2):      # twice: nothing kept from the first solve is in the way
        s.set_state(*st)
        code, _, lin = s.dev.newton(0.0)
        assert code == 0 and lin.converged and lin.iterations <= 30, (code, lin.iterations)
        got = np.concatenate(s.dev.get_state()[:2])
        d = np.linalg.norm(want - np.concatenate(st[:2]))
        assert np.linalg.norm(got - want) <= 1e-2 * d
    s.close()


def test_linear_system(v2d, oracle_mod):
    st, _ = far_state(v2d, oracle_mod)
    s = solver(v2d, oracle_mod, "fp64")
    s.set_state(*st)
    ip, ix, dv, b = s.dev.system(urot=0.0)
    s.close()
    n = b.size
    ci = np.repeat(np.arange(n, dtype=np.intc), np.diff(ip))
    lin = v2d.MumpsSolver(n, grid=(IMAX, JMAX), precision="mixed", max_it=60)
    for _ in range(2):
        lin.assemble(ci, ix, dv, b)
        x = lin.solve()     # raises unless the residual is below 1e-10 |b|
        r = b.copy()
        np.subtract.at(r, ci, dv * x[ix])
        assert np.linalg.norm(r) <= 2e-10 * np.linalg.norm(b)
    lin.destroy()


@pytest.mark.parametrize("cap", [15, 30, 100])
def test_batch_converges_where_fp64_does(v2d, oracle_mod, cap):
    """A sweep with instances whose Newton iteration diverges: whatever the limit
    of GMRES steps, the mixed batch converges on the instances FP64 does, to the
    same forces."""
    from vorti2d_b200.batch import Case, run_sweep_batched
    xg, yg = oracle_mod.generate_cylinder(IMAX, JMAX)
    cases = [Case(f"re{re:g}", xg, yg, re, 2.0)
             for re in (30.0, 60.0, 250.0, 400.0, 600.0, 900.0)]
    out = {p: run_sweep_batched(cases, precision=p, krylov_max_it=cap if p == "mixed" else 300)
           for p in ("fp64", "mixed")}
    a, b = ([r.converged for r in out[p].results] for p in ("fp64", "mixed"))
    assert a[0] and not all(a)
    assert a == b, (a, b)
    for x, y in zip(out["fp64"].results, out["mixed"].results):
        if x.converged:
            assert abs(x.cd - y.cd) <= 1e-8 and abs(x.cl - y.cl) <= 1e-8
