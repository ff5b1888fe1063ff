"""The pipelined linear solve (csrc/pipe_solve.cuh) of one domain in both step
schedules.  Its blocks each sum the last residual's partials after the solve's
last barrier and, in the fused step, go on to the Picard check, whose partials
must not be theirs.  Handles of a tile per block, and of several; iteration counts
long enough for solves to end in even and odd phases; against the launch-per-kernel
schedule, bit for bit."""
import numpy as np
import pytest

import dhara_b200 as db
from dhara_b200 import inputs

pytestmark = pytest.mark.gpu

FIELDS = ("psi", "theta", "ponding", "waterelev")


def run(d, fused, nsteps):
    s = db.Solver(d.params)
    s.load(d)
    s.prepare()
    c = s.launch_config()
    s.set_launch_config(c["krylov_blocks_per_sm"], c["overland_resident"], c["overland_blocks_per_sm"],
                        fused_step=fused)
    s.step(nsteps)
    s.synchronize()
    out = {k: s.download(k) for k in FIELDS}, s.diagnostics()
    s.close()
    return out


@pytest.mark.parametrize("prec", [db.FP64, db.MIXED])
@pytest.mark.parametrize("shape", [(19, 6, 3), (64, 60, 9), (160, 130, 6), (40, 33, 40)])
def test_one_domain_fused_equals_launch_per_kernel(gpu, shape, prec):
    d = inputs.make_domain(*shape, seed=9, precision=prec, rain_mm_per_h=30.0, nsteps=8, krylov_tol=1e-12,
                           krylov_maxiter=2000)
    (a, da), (b, dbg) = run(d, 0, 8), run(d, 1, 8)
    for k in FIELDS:
        assert np.array_equal(a[k], b[k]), k
    for k in ("picard_iters_total", "krylov_iters_total", "refine_iters_total", "krylov_nonconverged", "nonfinite"):
        assert da[k] == dbg[k], k
