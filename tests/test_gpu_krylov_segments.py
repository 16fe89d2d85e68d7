"""The captured pieces of a GMRES cycle, by the kernels launched: with kept FP64
factors they end at 1, 2, 4, 6, 8, 10, 14, 18, 22 and 30 steps, and at most one
piece past the cycle's last step is launched, or what the solve before took; with
fresh ones a solve of one step launches one."""
import numpy as np
import pytest

from cases import smooth_state

pytestmark = pytest.mark.gpu

STEP = 7          # scaling, LU solve, product, two passes of projection and update
BEGIN, END, TAIL = 2, 3, 1   # set-up and first residual; a cycle's end; the Newton update


def kept_launches(its, before):
    """At most: a piece that ends before `before` steps is followed by the next
    without a look; the cycle's end is queued behind steps 1 and 2 and once more."""
    ends = (1, 2, 4, 6, 8, 10, 14, 18, 22, 30)
    last = next(b for b in ends if b >= max(its, 2))
    looked = next(b for b in ends if b >= max(2, min(before - 1, 14)))
    return BEGIN + STEP * max(last, looked) + 3 * END + 2 * TAIL


def factorizations(v2d, s):
    out = np.zeros(6)
    v2d._lib.check(v2d._lib.lib().v2d_solver_phase_times(s.dev.h, v2d._lib.dptr(out), 0))
    return int(out[5])


def test_launches_with_kept_and_fresh_factors(v2d, oracle_mod):
    imax, jmax = 65, 49
    xg, yg = oracle_mod.generate_cylinder(imax, jmax)
    count = v2d._lib.lib().v2d_launch_count
    M = oracle_mod.core().compute_metrics(1 / (imax - 1), 1 / (jmax - 1), xg, yg)
    st = [np.array(a) for a in smooth_state(M[8], M[9])]
    seen = set()
    for rtol in (1e-2, 1e-4, 1e-6, 1e-8, 1e-10):
        s = v2d.Solver(v2d.Config(verbose=False, write_csv=False, write_xdmf=False, re=80.0,
                                  steady=False, dt_phys=0.2, ksp_restart=30, ksp_rtol=rtol,
                                  lu_reuse_its=30, lu_reuse_steps=True, precision="fp64"),
                       mesh=(xg, yg))
        s.set_state(*st)
        n0 = count()
        s.dev.system(urot=0.0)
        assembly = count() - n0
        code, _, lin = s.dev.newton(0.0)     # factors this Jacobian; captures the cycle
        assert code == 0 and lin.iterations == 1
        before = 0
        for amount in (1e-3, 1e-2, 1e-1):
            s.set_state(*[a * (1.0 + amount) for a in st])
            f0, n0 = factorizations(v2d, s), count()
            code, _, lin = s.dev.newton(0.0)
            assert code == 0 and lin.converged and factorizations(v2d, s) == f0
            got, most = count() - n0 - assembly, kept_launches(lin.iterations, before)
            assert got <= most, (rtol, before, lin.iterations)
            before = lin.iterations
            seen.add(lin.iterations)
        s.close()
    assert seen & {2, 5, 6, 9, 10}, seen     # where pieces of 1, 3, 4, 4 launched more
