"""The dataflow LU solve marks entries that are not computed yet with 0xff
bytes, which is a NaN: a matrix that holds this NaN ends like one with any
other, not by a wait that runs out."""
import numpy as np
import pytest

from cases import smooth_state

pytestmark = pytest.mark.gpu


def _status(v2d, n, ci, cj, cv, b):
    lin = v2d.MumpsSolver(n)
    try:
        lin.assemble(ci, cj, cv, b)
        return 0, lin.solve()
    except v2d._lib.V2DError as e:
        return e.code, None
    finally:
        lin.destroy()


@pytest.mark.parametrize("where", [0.1, 0.5, 0.9])
def test_nan_with_the_unset_pattern(v2d, oracle_mod, where):
    imax, jmax = 33, 29
    N, dk, de = imax * jmax, 1 / 32, 1 / 28
    M = oracle_mod.core().compute_metrics(dk, de, *oracle_mod.generate_cylinder(imax, jmax))
    st = smooth_state(M[8], M[9])
    ci, cj, cv, nnz, b = v2d.core.assemble_coo(imax, jmax, 80.0, 0.0, 2.5, 0.3, dk, de, *M, *st, 0,
                                               2 * N, 26 * N, 1, 1.0, 0.0)
    ci, cj, cv = ci[:nnz], cj[:nnz], cv[:nnz].copy()
    assert _status(v2d, 2 * N, ci, cj, cv, b)[0] == 0
    codes = []
    for bits in (0x7FF8000000000000, 0xFFFFFFFFFFFFFFFF):
        cv.view(np.uint64)[int(where * nnz)] = bits
        codes.append(_status(v2d, 2 * N, ci, cj, cv, b)[0])
    assert codes[0] == codes[1] != 0, codes
    assert codes[1] != v2d._lib.V2D_ETIMEOUT
