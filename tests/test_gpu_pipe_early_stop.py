"""A one-domain handle whose Picard iteration converges before its last allowed
iteration: the launch-per-kernel schedule queues the remaining solves all the same,
and these must leave the domain's record alone.  Against the same step with the
iterations it needs as the limit, where nothing is queued behind them: the same
state and the same report of the last solve, to the bit.  Loose solves and Picard
tolerances, where sums left over in the partials pass for a converged residual, and
a state at rest, where they are zero."""
import numpy as np
import pytest

import dhara_b200 as db
from dhara_b200 import inputs

pytestmark = pytest.mark.gpu

REPORT = ("picard_iters_total", "krylov_iters_total", "refine_iters_total", "krylov_nonconverged", "nonfinite",
          "krylov_relres_last", "picard_err_last")


def step(maxiter, prec, krylov_tol, rain, shape):
    d = inputs.make_domain(*shape, seed=4, precision=prec, rain_mm_per_h=rain, nsteps=1, krylov_tol=krylov_tol,
                           krylov_maxiter=2000, picard_rule=db.PICARD_PSI_ABSOLUTE, picard_tol=1e-2,
                           picard_maxiter=maxiter)
    st, dg, _ = db.run(d, nsteps=1)
    return st, dg


@pytest.mark.parametrize("prec", [db.FP64, db.MIXED])
@pytest.mark.parametrize("krylov_tol", [0.5, 1e-2, 1e-10])
@pytest.mark.parametrize("rain,shape", [(0.0, (24, 9, 5)), (30.0, (24, 9, 5)), (30.0, (64, 40, 12))])
def test_solves_after_convergence_change_nothing(gpu, rain, shape, krylov_tol, prec):
    a, da = step(20, prec, krylov_tol, rain, shape)
    used = da["picard_iters_total"]
    assert used < 20
    b, dbg = step(used, prec, krylov_tol, rain, shape)
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    for k in REPORT:
        assert da[k] == dbg[k], k
