"""Bounded waits of the LU factorization and solve: with their limits set so low
that they run out (at once, or somewhere along the way), the call ends
with V2D_ETIMEOUT, leaves the state alone and does not keep the factors; with the
default limits back, the same handle gives what an untouched one gives."""
import numpy as np
import pytest

from cases import smooth_state

pytestmark = pytest.mark.gpu


def solver(v2d, oracle_mod, n, **config):
    xg, yg = oracle_mod.generate_cylinder(n, n)
    s = v2d.Solver(v2d.Config(verbose=False, write_csv=False, write_xdmf=False, re=80.0,
                              steady=False, dt_phys=0.2, ksp_restart=30, **config), mesh=(xg, yg))
    M = oracle_mod.core().compute_metrics(1 / (n - 1), 1 / (n - 1), xg, yg)
    return s, smooth_state(M[8], M[9])


def limits(v2d, s, gather=-1, pipe=-1):
    v2d._lib.check(v2d._lib.lib().v2d_solver_lu_wait_limits(s.dev.h, gather, pipe))


def factorizations(v2d, s):
    out = np.zeros(6)
    v2d._lib.check(v2d._lib.lib().v2d_solver_phase_times(s.dev.h, v2d._lib.dptr(out), 0))
    return int(out[5])


# 181 x 181: levels wide enough for the pipelined update in FP64
@pytest.mark.parametrize("n,precision,form,split,reuse", [
    (181, "fp64", 0, 0, 0), (181, "fp64", 1, 0, 0), (181, "fp64", 0, 4, 8), (65, "fp64", 0, 0, 8),
    (181, "mixed", 0, 0, 0), (97, "mixed", 1, 3, 8)])
def test_waits_that_run_out(v2d, oracle_mod, n, precision, form, split, reuse):
    s, st = solver(v2d, oracle_mod, n, precision=precision, lu_reuse_its=reuse,
                   lu_reuse_steps=True)
    L = v2d._lib.lib()
    s.set_state(*st)
    assert s.dev.newton(0.0)[0] == 0
    v2d._lib.check(L.v2d_solver_lu_flow_form(s.dev.h, form, None))
    v2d._lib.check(L.v2d_solver_lu_split(s.dev.h, split, None))
    s.set_state(*st)
    code, res, lin = s.dev.newton(0.0)
    assert code == 0 and lin.converged
    want = s.dev.get_state()
    for gather, pipe in [(0, -1), (-1, 0), (-1, 1), (-1, 5), (-1, 40), (3, 200)]:
        limits(v2d, s, gather, pipe)
        s.set_state(*st)
        f0 = factorizations(v2d, s)
        code, _, _ = s.dev.newton(0.0)
        if gather == 0 or pipe == 0:
            assert code == v2d._lib.V2D_ETIMEOUT, (gather, pipe, code)
        assert code in (0, v2d._lib.V2D_ETIMEOUT), (gather, pipe, code)
        if code != 0:
            assert "timed out" in v2d._lib.last_error()
            if precision == "fp64" and n == 181 and reuse == 0 and pipe == 0:
                assert "LU factor" in v2d._lib.last_error()
            for a, b in zip(s.dev.get_state(), st):
                assert np.array_equal(a, b)      # no update
        limits(v2d, s)
        s.set_state(*st)
        f1 = factorizations(v2d, s)
        again, _, lin = s.dev.newton(0.0)
        assert again == 0 and lin.converged
        if code != 0:
            assert factorizations(v2d, s) == f1 + 1 and f1 >= f0    # the old ones were dropped
        if reuse == 0:   # (kept factors of another solve: the same to the tolerance only)
            for a, b in zip(s.dev.get_state()[:2], want[:2]):
                assert np.array_equal(a, b)
    s.close()


def test_adjoint_reports_a_factorization_that_gave_up(v2d, oracle_mod):
    from vorti2d_b200.adjoint import adjoint_solve
    s, st = solver(v2d, oracle_mod, 181, precision="fp64")
    s.set_state(*st)
    assert s.dev.newton(0.0)[0] == 0
    g = np.random.default_rng(3).standard_normal(2 * s.ndof)
    lam, its, rel = adjoint_solve(s, g, rtol=1e-10)
    limits(v2d, s, -1, 0)
    s.set_state(*st)
    with pytest.raises(v2d._lib.V2DError) as e:
        adjoint_solve(s, g, rtol=1e-10)
    assert e.value.code == v2d._lib.V2D_ETIMEOUT
    limits(v2d, s)
    lam2, _, rel = adjoint_solve(s, g, rtol=1e-10)   # not the factors that were given up
    assert rel <= 2e-10
    s.close()
