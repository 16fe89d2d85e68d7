"""The Newton update is queued behind the Krylov solve, gated on the device:
what a failed assembly, an unconverged and a converged solve leave behind."""
import numpy as np
import pytest

from cases import smooth_state

pytestmark = pytest.mark.gpu


def _solver(v2d, oracle_mod, **config):
    imax, jmax = 33, 29
    xg, yg = oracle_mod.generate_cylinder(imax, jmax)
    s = v2d.Solver(v2d.Config(verbose=False, write_csv=False, write_xdmf=False, re=80.0,
                              steady=False, dt_phys=0.2, ksp_restart=30, **config), mesh=(xg, yg))
    M = oracle_mod.core().compute_metrics(1 / (imax - 1), 1 / (jmax - 1), xg, yg)
    return s, smooth_state(M[8], M[9])


@pytest.mark.parametrize("precision,reuse", [("fp64", 0), ("mixed", 0), ("mixed", 8)])
def test_non_finite_state_is_reported_and_left_alone(v2d, oracle_mod, precision, reuse):
    s, st = _solver(v2d, oracle_mod, precision=precision, lu_reuse_its=reuse)
    s.set_state(*st)
    code, res, lin = s.dev.newton(0.0)
    assert code == 0 and lin.converged
    want = np.concatenate(s.dev.get_state()[:2])
    bad = [a.copy() for a in st]
    bad[1][100] = np.nan
    s.set_state(*bad)
    code, _, _ = s.dev.newton(0.0)
    assert code == -4 and "newton assembly" in v2d._lib.last_error()
    after = s.dev.get_state()
    for a, b in zip(after[:2], bad[:2]):
        assert np.array_equal(a, b, equal_nan=True)   # no update
    s.set_state(*st)
    code, res2, lin = s.dev.newton(0.0)
    assert code == 0 and lin.converged
    # both solves stop below rtol (1e-5 or tighter) times the same residual
    got = np.concatenate(s.dev.get_state()[:2])
    assert np.max(np.abs(got - want)) <= 1e-3 * np.max(np.abs(want - np.concatenate(st[:2])))
    s.close()


def test_unconverged_solve_updates_once_and_says_so(v2d, oracle_mod):
    s, st = _solver(v2d, oracle_mod, precision="mixed", krylov_max_it=1, ksp_rtol=1e-14)
    s.set_state(*st)
    code, res, lin = s.dev.newton(0.0)
    assert code == -5 and not lin.converged and lin.iterations == 1
    # the norm is that of the one update that was applied
    d = np.concatenate(s.dev.get_state()[:2]) - np.concatenate(st[:2])
    assert np.isclose(np.linalg.norm(d) / d.size, res, rtol=1e-6)
    s.close()
