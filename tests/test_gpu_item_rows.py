"""The solve's work items after a change of one level's rows: the other levels
keep theirs, the separate backward rows of the default split among them."""
import ctypes

import numpy as np
import pytest

from cases import smooth_state

pytestmark = pytest.mark.gpu


def trace_items(v2d, s):
    L, ip = v2d._lib.lib(), v2d._lib.iptr
    cap = 200000
    items, ticks, n = np.zeros(12 * cap, dtype=np.intc), (ctypes.c_ulonglong * (3 * cap))(), ctypes.c_int()
    v2d._lib.check(L.v2d_solver_trace_lu_apply(s.dev.h, ticks, ip(items), cap, ctypes.byref(n)))
    return items[:12 * n.value].reshape(-1, 12).copy()


def of_level(items, L, kind):
    it = items[(items[:, 10] == L) & (items[:, 0] == kind)]
    return [tuple(int(v) for v in r[1:4]) for r in it]


def test_one_level_changes_alone(v2d, oracle_mod):
    from vorti2d_b200 import tune
    imax = jmax = 181
    xg, yg = oracle_mod.generate_cylinder(imax, jmax)
    M = oracle_mod.core().compute_metrics(1 / (imax - 1), 1 / (jmax - 1), xg, yg)
    s = v2d.Solver(v2d.Config(verbose=False, write_csv=False, write_xdmf=False, re=80.0,
                              steady=False, dt_phys=0.2, ksp_restart=30), mesh=(xg, yg))
    s.set_state(*smooth_state(M[8], M[9]))
    assert s.dev.newton(0.0)[0] == 0
    start, rows = trace_items(v2d, s), tune.item_rows(s)
    nl = len(rows)

    def span(items, L, kind):
        return max(b - a for _, a, b in of_level(items, L, kind))

    split = [L for L in range(nl) if rows[L] > 0 and span(start, L, 1) < min(
        rows[L], span(start, L, 0))]
    assert split     # levels with fewer rows per backward item
    for L in (split[0], nl - 1):
        trial = list(rows)
        trial[L] = 8 if rows[L] != 8 else 16
        tune.set_item_rows(s, trial)
        now = trace_items(v2d, s)
        assert tune.item_rows(s) == trial
        for K in range(nl):
            for kind in (0, 1):
                if K != L:
                    assert of_level(now, K, kind) == of_level(start, K, kind), (L, K, kind)
                else:
                    assert span(now, K, kind) <= trial[L]
    tune.set_item_rows(s, rows)
    assert np.array_equal(trace_items(v2d, s), start)
    s.close()
