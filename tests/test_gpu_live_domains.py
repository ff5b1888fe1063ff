"""The 3D solve of many domains that stop at very different iterations: most blocks
have no tile of the last ones and only follow the count of live domains from barrier
to barrier (kry_live, csrc/device_common.cuh).  A loose tolerance for all domains but
a few, which last long after; the batch against the long ones alone, and against
itself, bit for bit, and their iteration counts."""
import numpy as np
import pytest

import dhara_b200 as db
from dhara_b200 import inputs

pytestmark = pytest.mark.gpu

COUNTS = ("picard_iters_total", "krylov_iters_total", "refine_iters_total", "krylov_nonconverged")


@pytest.mark.parametrize("prec", [db.FP64, db.MIXED])
@pytest.mark.parametrize("last", [(0,), (149,), (3, 77, 148)])
def test_few_domains_outlast_the_rest(gpu, last, prec):
    doms = [inputs.make_domain(16 + i % 9, 5 + i % 3, 4 + i % 7, seed=i, precision=prec, rain_mm_per_h=30.0, nsteps=3,
                               krylov_tol=1e-13 if i in last else 1e-2, krylov_maxiter=2000) for i in range(150)]
    a, b = db.run(doms), db.run(doms)
    for i in range(len(doms)):
        for k in a[i][0]:
            assert np.array_equal(a[i][0][k], b[i][0][k]), (i, k)
    for i in last:
        one, dg, _ = db.run(doms[i])
        for k in one:
            assert np.array_equal(a[i][0][k], one[k]), (i, k)
        for k in COUNTS:
            assert a[i][1][k] == dg[k], (i, k)
    assert min(a[i][1]["krylov_iters_total"] for i in last) > max(
        a[i][1]["krylov_iters_total"] for i in range(len(doms)) if i not in last)
