"""The pipelined linear solve where its two kinds of sweep lay out a block's shared
memory differently: with several tiles per block, FP64 columns of 26 to 35 layers
have two column buffers in phase R and one in the inner sweeps, mixed columns of 48
and 49 layers the other way round, so that what warps write as a column buffer in
one sweep is written by the TMA as a stage in the next.  Both edges of each range
and the heights beside them: every domain of a batch of several tiles per block
against the domain alone (a tile per block, one buffer in both), bit for bit."""
import numpy as np
import pytest

import dhara_b200 as db
from dhara_b200 import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,nz", [(db.FP64, 25), (db.FP64, 26), (db.FP64, 30), (db.FP64, 35), (db.FP64, 36),
                                     (db.MIXED, 47), (db.MIXED, 48), (db.MIXED, 49), (db.MIXED, 50)])
def test_unequal_column_buffers(gpu, prec, nz):
    # 3 tiles each (16 x 8): 234 tiles, one or two for each of the GPU's 148 SMs
    doms = [inputs.make_domain(37 + i % 3, 8, nz, seed=i, precision=prec, krylov_tol=1e-12, krylov_maxiter=2000,
                               nsteps=2, rain_mm_per_h=30.0) for i in range(78)]
    batch = db.run(doms, nsteps=2)
    for i in (0, 1, 2, 38, 75, 76, 77):
        one, dg, _ = db.run(doms[i], nsteps=2)
        for k in one:
            assert np.array_equal(batch[i][0][k], one[k]), (i, k)
        assert batch[i][1]["krylov_iters_total"] == dg["krylov_iters_total"], i
