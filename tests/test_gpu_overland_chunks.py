"""The overland multigrid solve over the sizes of its level-0 chunks (one, two or
four groups of 512 points by the handle's points, csrc/overland_mg.cu): a
surface's solve is the same bits whichever size its handle takes, and agrees with
the Jacobi solver's to the tolerance both converge to (as in test_gpu_overland_mg).
The sizes: interiors of 511, 512 and 513 points, one past the block levels
(36 x 36), and handles of 161 and 314 groups, where the chunk grows."""
import numpy as np
import pytest

import dhara_b200 as db
from dhara_b200 import inputs

pytestmark = pytest.mark.gpu

SIZES = [(9, 75), (34, 18), (29, 21), (38, 38), (61, 47)]  # interiors 511, 512, 513, 1296, 2655


def surface(nx, ny, solver=0):
    d = inputs.make_domain(nx, ny, 2, seed=nx + ny, precision=db.FP64, nsteps=1, overland_tol=1e-12,
                           overland_maxiter=20000, overland_solver=solver)
    r = np.random.default_rng(nx * ny)
    return d, 2e-3 * r.random(nx * ny)


def solve(items):
    s = db.Solver([d.params for d, _ in items])
    for i, (d, _) in enumerate(items):
        s.load(d, i)
    s.prepare()
    for i, (_, depth) in enumerate(items):
        s.upload("waterdepth", depth, i)
    s.overland_step()
    s.synchronize()
    out = [(s.download("waterelev", i), s.diagnostics(i)) for i in range(len(items))]
    s.close()
    return out


@pytest.mark.parametrize("extra", [(280, 274), (400, 389)], ids=["two_groups", "four_groups"])
def test_chunk_sizes_same_bits(gpu, extra):
    items = [surface(*n) for n in SIZES + [extra]]
    batch = solve(items)
    for it, (h, dg) in zip(items[:len(SIZES)], batch):
        (one, od), = solve([it])
        assert np.array_equal(h, one), (it[0].params.nx, it[0].params.ny)
        assert dg["overland_iters_total"] == od["overland_iters_total"] and dg["overland_nonconverged"] == 0


@pytest.mark.parametrize("size", SIZES)
def test_against_jacobi(gpu, size):
    (a, da), = solve([surface(*size)])
    (b, dbg), = solve([surface(*size, solver=1)])
    assert da["overland_nonconverged"] == 0 and dbg["overland_nonconverged"] == 0
    assert np.max(np.abs(a - b)) < 1e-9 * np.max(np.abs(b))
