"""The transposed solve's shared memory: a grid whose fronts need more than a
launch has without raising the limit."""
import numpy as np
import pytest
import scipy.sparse as sp

from cases import smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("imax,jmax", [(1601, 9), (1601, 12)])
def test_transposed_solve_of_wide_fronts(v2d, oracle_mod, imax, jmax):
    """1601 columns: fronts of 3202 and more unknowns, over 50 KB for the two
    vectors of a front in FP64 (48 KB without a raised limit).  GMRES stops at
    1e-10 of its own FP64 residual: within twice that here."""
    from vorti2d_b200.adjoint import adjoint_solve
    xg, yg = oracle_mod.generate_cylinder(imax, jmax)
    s = v2d.Solver(v2d.Config(verbose=False, write_csv=False, write_xdmf=False,
                              compute_forces=False, re=80.0, steady=False, dt_phys=0.05),
                   mesh=(xg, yg))
    M = oracle_mod.core().compute_metrics(1 / (imax - 1), 1 / (jmax - 1), xg, yg)
    s.set_state(*smooth_state(M[8], M[9]))
    g = np.random.default_rng(2).standard_normal(2 * s.ndof)
    lam, its, rel = adjoint_solve(s, g, rtol=1e-10)
    ip, ix, dv, _ = s.dev.system(urot=0.0)
    J = sp.csr_matrix((dv, ix, ip), shape=(2 * s.ndof, 2 * s.ndof))
    assert np.linalg.norm(J.T @ lam - g) <= 2e-10 * np.linalg.norm(g), (its, rel)
    s.close()
