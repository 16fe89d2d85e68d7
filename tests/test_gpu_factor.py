"""The block Gauss-Jordan elimination of the fronts (64 pivots per step, two
32-wide halves in the pivot block, 64 x 64 tiles) at the widths where a step,
a half or a tile ends: the root separator of an imax x jmax O-grid has
2 imax pivots and no contribution rows, its children 4 (jmax/2) pivots.

Tolerances: the update is compared at 1e-9 like every one-update test.  FP64
factors with row-scaled 64-row pivot blocks have a backward error of about
n eps times the element growth (n <= 1e4, eps = 1.1e-16, growth at most 1e3
assumed: 1e-9), so two GMRES iterations reach 1e-12; FP32 factors (eps = 6e-8,
the same n times growth taken as 1e5) reduce the residual by 1e-2 at least per
iteration: six reach 1e-12.  One more is allowed to each."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from cases import smooth_state

pytestmark = pytest.mark.gpu

# root widths 30, 32, 34, 62, 64, 66, 96, 98, 126, 128, 130, 254, 258
WIDTHS = [(15, 13), (16, 13), (17, 13), (31, 17), (32, 17), (33, 17), (48, 33), (49, 33), (63, 31),
          (64, 32), (65, 33), (127, 64), (129, 67)]


def one_update(v2d, oracle_mod, imax, jmax, limit, tol=1e-9, **config):
    """One Newton update on an imax x jmax grid against SciPy's direct solve, refined."""
    xg, yg = oracle_mod.generate_cylinder(imax, jmax)
    s = v2d.Solver(v2d.Config(verbose=False, write_csv=False, write_xdmf=False, re=80.0,
                              steady=False, dt_phys=0.2, farfield_bc="outflow", alpha_deg=4.0,
                              ksp_rtol=1e-12, ksp_restart=30, **config), mesh=(xg, yg))
    M = oracle_mod.core().compute_metrics(1 / (imax - 1), 1 / (jmax - 1), xg, yg)
    st = smooth_state(M[8], M[9])
    s.set_state(*st)
    N = imax * jmax
    ci, cj, cv, nnz, b = oracle_mod.core().assemble_coo(
        imax, jmax, 80.0, 0.0, 2.5, 0.3, 1 / (imax - 1), 1 / (jmax - 1), *M, *st, 0, 2 * N,
        26 * N, 1, np.cos(np.radians(4.0)), np.sin(np.radians(4.0)))
    A = sp.csr_matrix((cv[:nnz], (ci[:nnz], cj[:nnz])), shape=(2 * N, 2 * N))
    lu = spla.splu(A.tocsc())
    dq = lu.solve(b)
    dq += lu.solve(b - A @ dq)   # refined: the direct solve alone is 3e-6 off at 257 x 257
    code, _, lin = s.dev.newton(0.3)
    assert code == 0, v2d._lib.last_error()
    got = np.concatenate(s.dev.get_state()[:2]) - np.concatenate(st[:2])
    s.close()
    assert np.max(np.abs(got - dq)) <= tol * max(1.0, np.max(np.abs(dq)))
    assert lin.converged and lin.iterations <= limit, lin.iterations


@pytest.mark.parametrize("imax,jmax", WIDTHS)
@pytest.mark.parametrize("precision,factors,limit", [("fp64", "fp32", 3), ("mixed", "fp32", 7),
                                                     ("mixed", "fp64", 7)])
def test_elimination_widths(v2d, oracle_mod, imax, jmax, precision, factors, limit):
    one_update(v2d, oracle_mod, imax, jmax, limit, precision=precision, lu_factors=factors)


# The leaf kernel's blocks of 32 and 8 pivots (at most 128 = 64 nodes) and the
# leaves beyond it, eliminated like the other fronts; the whole grid one leaf
@pytest.mark.parametrize("leaf,imax,jmax", [(4, 23, 19), (9, 23, 19), (16, 33, 33), (17, 33, 29),
                                            (33, 41, 27), (48, 41, 35), (63, 63, 31), (64, 33, 33),
                                            (64, 8, 8), (65, 33, 33), (100, 37, 33), (512, 16, 16)])
@pytest.mark.parametrize("precision,factors,limit", [("fp64", "fp32", 3), ("mixed", "fp32", 7),
                                                     ("mixed", "fp64", 7)])
def test_leaf_sizes(v2d, oracle_mod, monkeypatch, leaf, imax, jmax, precision, factors, limit):
    defaults = v2d._lib.krylov_defaults

    def with_leaf():   # a parameter of the C interface only
        k = defaults()
        k.lu_leaf = leaf
        return k

    monkeypatch.setattr(v2d._lib, "krylov_defaults", with_leaf)
    one_update(v2d, oracle_mod, imax, jmax, limit, precision=precision, lu_factors=factors)


# Levels wide enough for the pipelined update (592 tiles of fronts with 64
# pivots or more): fronts of different sizes with a part step after the full
# one (78 to 90 pivots), of exactly one step (64), of three full steps and a
# part (254, 256).  The update's error grows with the condition, here up to
# eight times the nodes and so at most ten times that of the grids above: 1e-8.
@pytest.mark.parametrize("imax,jmax", [(181, 181), (193, 161), (513, 33), (257, 257)])
@pytest.mark.parametrize("precision,factors,limit", [("fp64", "fp32", 3), ("mixed", "fp64", 7)])
def test_wide_update(v2d, oracle_mod, imax, jmax, precision, factors, limit):
    one_update(v2d, oracle_mod, imax, jmax, limit, tol=1e-8, precision=precision,
               lu_factors=factors)
