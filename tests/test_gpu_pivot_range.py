"""The pivots' reciprocals over the FP64 range, and subnormal pivots in the fronts'
elimination: one whose reciprocal is finite is one like any other.

The elimination's matrix is the identity on the O-grid's pattern but for one row, whose
diagonal entry is the pivot and which holds a one in another column, so that the
row scaling leaves it; with b = A x, x = 1 and 0 in that column, every product is
exact up to the pivot's own reciprocal: a few units in the last place."""
import numpy as np
import pytest

from cases import smooth_state

pytestmark = pytest.mark.gpu


def test_reciprocals(v2d):
    """Within 2 units in the last place (2^-52 relative at most, each) of 1 / x,
    which NumPy rounds correctly; where 1 / x is subnormal, within one unit of
    those, and infinite where it is."""
    rng = np.random.default_rng(7)
    n = 400000
    e = np.concatenate([rng.integers(-1024, 1024, n - 20000), rng.integers(-1024, -1018, 10000),
                        rng.integers(1017, 1024, 10000)])
    x = np.ldexp(rng.uniform(1.0, 2.0, n), e) * rng.choice([-1.0, 1.0], n)
    x[:10000] = np.ldexp(1.0, e[:10000])                                   # powers of two
    x[10000:20000] = np.nextafter(np.ldexp(1.0, e[10000:20000]), 0.0)      # and just below
    x = np.concatenate([x, [5e-324, 2.0 ** -1022, 2.0 ** -1021, 2.0 ** 1021, 2.0 ** 1023,
                            np.finfo(float).max]])
    y = np.empty_like(x)
    v2d._lib.check(v2d._lib.lib().v2d_lu_reciprocals(x.size, v2d._lib.dptr(x), v2d._lib.dptr(y)))
    with np.errstate(all="ignore"):
        want = 1.0 / x
    tiny, inf = np.abs(want) < 2.0 ** -1022, np.isinf(want)
    assert np.array_equal(y[inf], want[inf])
    assert np.max(np.abs(y[tiny] - want[tiny])) <= 5e-324
    rest = ~(tiny | inf)
    assert np.max(np.abs(y[rest] / want[rest] - 1.0)) <= 2 * 2.0 ** -52


# 2^-1022 is the smallest normal number, 2^-1023 and 1.5 * 2^-1024 are subnormal
# (reciprocals up to 1.2e308)
@pytest.mark.parametrize("pivot", [2.0 ** 0, 2.0 ** -500, 2.0 ** -1022, 2.0 ** -1023,
                                   1.5 * 2.0 ** -1024])
# a node of a leaf, one of the root separator (jmax / 2)
@pytest.mark.parametrize("node", [(3, 2), (10, 14)])
def test_small_pivots(v2d, oracle_mod, pivot, node):
    imax, jmax = 33, 29
    N, dk, de = imax * jmax, 1 / 32, 1 / 28
    M = oracle_mod.core().compute_metrics(dk, de, *oracle_mod.generate_cylinder(imax, jmax))
    ci, cj, cv, nnz, _ = v2d.core.assemble_coo(imax, jmax, 80.0, 0.0, 2.5, 0.3, dk, de, *M,
                                               *smooth_state(M[8], M[9]), 0, 2 * N, 26 * N, 1,
                                               1.0, 0.0)
    ci, cj = ci[:nnz], cj[:nnz]
    cv = (ci == cj).astype(float)
    r = N + node[1] * imax + node[0]            # the node's vorticity row ...
    c = r + 1                                   # ... couples to the next node's
    assert ((ci == r) & (cj == c)).sum() == 1
    cv[(ci == r) & (cj == r)] = pivot
    cv[(ci == r) & (cj == c)] = 1.0
    x = np.ones(2 * N)
    x[c] = 0.0
    b = np.zeros(2 * N)
    np.add.at(b, ci, cv * x[cj])
    lin = v2d.MumpsSolver(2 * N, grid=(imax, jmax), rtol=1e-12)
    lin.assemble(ci, cj, cv, b)
    got = lin.solve()
    lin.destroy()
    assert np.max(np.abs(got - x)) <= 1e-14, np.max(np.abs(got - x))
