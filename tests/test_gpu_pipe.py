"""The pipelined linear solve (csrc/pipe_solve.cuh) at the edges of its shapes:
one plane, a unit and a half, the tallest columns it takes and the first it
leaves to krylov_solve (FP64 columns of over 48 layers), widths that fill no
tile, and blocks with several tiles of several domains, with one and with two
column buffers.  Against the FP64 oracle with the parity tests' tolerances
(FP64 1e-8 and mixed 1e-6 for solves to 1e-12), and a batch against its domains
run alone, bit for bit."""
import numpy as np
import pytest

import dhara_b200 as db
from dhara_b200 import inputs
import oracle

from conftest import rel_err

pytestmark = pytest.mark.gpu


def domain(nx, ny, nz, prec, seed=5):
    return inputs.make_domain(nx, ny, nz, seed=seed, precision=prec, krylov_tol=1e-12, krylov_maxiter=2000, nsteps=2,
                              rain_mm_per_h=30.0)


@pytest.mark.parametrize("shape,prec", [((19, 6, 1), db.FP64), ((33, 5, 3), db.MIXED), ((31, 9, 48), db.FP64),
                                        ((31, 9, 49), db.FP64), ((31, 9, 64), db.MIXED), ((45, 50, 5), db.FP64)])
def test_column_heights(gpu, shape, prec):
    d = domain(*shape, prec)
    g, _, _ = db.run(d, nsteps=1)
    o, _, _ = oracle.run(d, nsteps=1, solver3d=oracle.SOLVER_CG)
    for k in ("psi", "theta", "waterelev"):
        assert rel_err(g[k], o[k]) < (1e-8 if prec == db.FP64 else 1e-6), (k, shape)


@pytest.mark.parametrize("prec,ndom,nz", [(db.FP64, 110, 7), (db.FP64, 110, 45), (db.MIXED, 190, 9), (db.MIXED, 190, 63)])
def test_several_tiles_per_block(gpu, prec, ndom, nz):
    # 2 to 4 tiles a domain, up to 3 (FP64) or 4 per SM: above that FP64 handles of
    # several domains run krylov_solve, whose sums have another order
    doms = [domain(17 + 5 * (i % 4), 7 + i % 9, max(2, nz - i % 5), prec, seed=i) for i in range(ndom)]
    batch = db.run(doms, nsteps=1)
    for i in (0, 77, ndom - 1):
        one, od, _ = db.run(doms[i], nsteps=1)
        for k in one:
            assert np.array_equal(batch[i][0][k], one[k]), (i, k)
        o, _, _ = oracle.run(doms[i], nsteps=1, solver3d=oracle.SOLVER_CG)
        for k in ("psi", "theta", "waterelev"):
            assert rel_err(one[k], o[k]) < (1e-8 if prec == db.FP64 else 1e-6), (i, k)
