"""The first solve of a linear system with kept factors asked for: it factors the
matrix, it does not try factors that were never made."""
import numpy as np
import pytest

from cases import smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_first_solve_factors(v2d, oracle_mod, precision):
    imax, jmax = 33, 29
    N, dk, de = imax * jmax, 1 / 32, 1 / 28
    M = oracle_mod.core().compute_metrics(dk, de, *oracle_mod.generate_cylinder(imax, jmax))
    ci, cj, cv, nnz, b = v2d.core.assemble_coo(imax, jmax, 80.0, 0.0, 2.5, 0.3, dk, de, *M,
                                               *smooth_state(M[8], M[9]), 0, 2 * N, 26 * N, 1,
                                               1.0, 0.0)
    got = []
    for reuse in (0, 8):
        lin = v2d.MumpsSolver(2 * N, precision=precision, lu_reuse_its=reuse)
        lin.assemble(ci[:nnz], cj[:nnz], cv[:nnz], b)
        x = lin.solve()
        got.append((lin.last_stats.iterations, x))
        lin.assemble(ci[:nnz], cj[:nnz], 1.001 * cv[:nnz], b)
        y = lin.solve()      # the second may keep them
        assert np.max(np.abs(1.001 * y - x)) <= 1e-6 * np.max(np.abs(x))
        lin.destroy()
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
