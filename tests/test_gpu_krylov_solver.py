"""The two solvers of the 3D system, chosen by dhara_launch_config.krylov_solver:
krylov_solve, which large handles take, at the small and ragged sizes where it can go
wrong (against the oracle with the parity tests' tolerances for solves to 1e-12, FP64
1e-8 and mixed 1e-6; with Dirichlet faces as in test_gpu_dirichlet), its independence
of block counts and step schedules, bit for bit, and of the other domains of a batch;
which solver a handle takes and reports, by itself and when asked; and that the
tuner does not choose among block counts the pipeline does not have."""
import numpy as np
import pytest

import dhara_b200 as db
from dhara_b200 import inputs
import oracle

from conftest import rel_err
from test_gpu_dirichlet import domain_with_faces

pytestmark = pytest.mark.gpu

PIPELINE, BLOCKS = 1, 2
FIELDS = ("psi", "theta", "ponding", "waterelev")


def solver(doms, choose=None, per_sm=None, **kw):
    doms = doms if isinstance(doms, list) else [doms]
    s = db.Solver([d.params for d in doms])
    for i, d in enumerate(doms):
        s.load(d, i)
    s.prepare()
    c = s.launch_config()
    s.set_launch_config(per_sm or c["krylov_blocks_per_sm"], c["overland_resident"], c["overland_blocks_per_sm"],
                        krylov_solver=choose, **kw)
    return s


def run(doms, choose, nsteps=1, per_sm=None, **kw):
    with solver(doms, choose, per_sm, **kw) as s:
        assert choose is None or s.launch_config()["krylov_solver"] == choose
        s.step(nsteps)
        s.synchronize()
        n = len(doms) if isinstance(doms, list) else 1
        return [({k: s.download(k, i) for k in FIELDS}, s.diagnostics(i)) for i in range(n)]


def domain(nx, ny, nz, prec, seed=5, nsteps=2):
    return inputs.make_domain(nx, ny, nz, seed=seed, precision=prec, krylov_tol=1e-12, krylov_maxiter=2000,
                              nsteps=nsteps, rain_mm_per_h=30.0)


def same(a, b):
    for (sa, da), (sb, dbg) in zip(a, b):
        for k in FIELDS:
            assert np.array_equal(sa[k], sb[k]), k
        for k in ("picard_iters_total", "krylov_iters_total", "refine_iters_total"):
            assert da[k] == dbg[k], k


@pytest.mark.parametrize("prec", [db.FP64, db.MIXED])
@pytest.mark.parametrize("shape", [(19, 6, 1), (33, 5, 3), (31, 9, 48), (31, 9, 64), (45, 50, 5), (5, 70, 4)])
def test_blocks_match_oracle_at_small_sizes(gpu, shape, prec):
    d = domain(*shape, prec)
    (g, _), = run(d, BLOCKS)
    o, _, _ = oracle.run(d, nsteps=1, solver3d=oracle.SOLVER_CG)
    for k in ("psi", "theta", "waterelev"):
        assert rel_err(g[k], o[k]) < (1e-8 if prec == db.FP64 else 1e-6), k


@pytest.mark.parametrize("prec", [db.FP64, db.MIXED])
@pytest.mark.parametrize("choose", [PIPELINE, BLOCKS])
def test_dirichlet_faces(gpu, choose, prec):
    d = domain_with_faces({"south": -0.4, "west": -0.3, "bottom": 0.1}, prec=prec)
    o, _, _ = oracle.run(d, nsteps=3, solver3d=oracle.SOLVER_BICGSTAB)
    a, b = run(d, choose, 3, fused_step=0), run(d, choose, 3, fused_step=1)
    same(a, b)
    for k in ("psi", "theta", "ponding"):
        assert rel_err(a[0][0][k], o[k]) < 1e-6, k


@pytest.mark.parametrize("prec", [db.FP64, db.MIXED])
def test_blocks_do_not_depend_on_count_or_schedule(gpu, prec):
    # the second batch has more tiles (402) than the smallest grid has blocks
    for doms in ([domain(40, 36, 12, prec)], [domain(17 + 5 * (i % 4), 7 + i % 9, 3 + i % 5, prec, i) for i in range(150)]):
        base = run(doms, BLOCKS, 2, fused_step=0)
        with solver(doms) as s:
            most = s.launch_config()["krylov_blocks_per_sm"]
        for per_sm in range(1, most + 1):
            same(base, run(doms, BLOCKS, 2, per_sm, fused_step=per_sm % 2))


@pytest.mark.parametrize("prec", [db.FP64, db.MIXED])
@pytest.mark.parametrize("last", [(0,), (149,), (3, 77, 148)])
def test_blocks_when_few_domains_outlast_the_rest(gpu, last, prec):
    doms = [inputs.make_domain(16 + i % 9, 5 + i % 3, 4 + i % 7, seed=i, precision=prec, rain_mm_per_h=30.0, nsteps=3,
                               krylov_tol=1e-13 if i in last else 1e-2, krylov_maxiter=2000) for i in range(150)]
    a = run(doms, BLOCKS, 3)
    for i in last:
        same([a[i]], run(doms[i], BLOCKS, 3))


@pytest.mark.parametrize("prec,nz,fits", [(db.FP64, 50, True), (db.FP64, 51, False), (db.FP64, 64, False),
                                          (db.MIXED, 64, True)])
def test_tallest_columns_of_the_pipeline(gpu, prec, nz, fits):
    """The first FP64 column too tall for the pipeline has 51 layers."""
    d = domain(31, 9, nz, prec)
    with solver(d) as s:
        assert s.launch_config()["krylov_solver"] == (PIPELINE if fits else BLOCKS)
    with solver(d, PIPELINE) as s:
        assert s.launch_config()["krylov_solver"] == (PIPELINE if fits else BLOCKS)
        s.step(1)
        s.synchronize()
        got = {k: s.download(k) for k in FIELDS}
    (want, _), = run(d, BLOCKS)
    for k in ("psi", "theta", "waterelev"):
        assert rel_err(got[k], want[k]) < (1e-8 if prec == db.FP64 else 1e-6), k


def test_choice_follows_the_tile_shape(gpu):
    """16 x 3600 FP64 columns: 450 tiles of 16 x 8 (4 per SM in one round of
    krylov_solve's blocks, which it keeps), 900 of 32 x 4 (7 in two rounds)."""
    d = domain(16, 3600, 2, db.FP64)
    with solver(d) as s:
        c = s.launch_config()

        def shape(t, choose=None):
            s.set_launch_config(c["krylov_blocks_per_sm"], c["overland_resident"], c["overland_blocks_per_sm"], t,
                                krylov_solver=choose)
            return s.launch_config()["krylov_solver"]
        assert c["krylov_solver"] == BLOCKS
        assert [shape(1), shape(2), shape(1)] == [PIPELINE, BLOCKS, PIPELINE]
        # asked for, it stays; 0 goes back to the rule
        assert [shape(1, BLOCKS), shape(2), shape(1), shape(1, 0), shape(2, PIPELINE), shape(2, 0)] == \
            [BLOCKS, BLOCKS, BLOCKS, PIPELINE, PIPELINE, BLOCKS]
        s.step(1)
        s.synchronize()
        assert s.diagnostics()["nonfinite"] == 0


@pytest.mark.parametrize("choose", [PIPELINE, BLOCKS])
def test_autotune_keeps_the_solver(gpu, choose):
    with solver(domain(40, 36, 12, db.MIXED, nsteps=8), choose, per_sm=2) as s:
        n0 = s.launch_count()
        got = s.autotune(1)
        assert got["krylov_solver"] == choose == s.launch_config()["krylov_solver"]
        assert got["krylov_ms"] > 0
        if choose == PIPELINE:  # has no block counts to choose from
            assert got["krylov_blocks_per_sm"] == 2
        assert s.launch_count() == n0
        s.step(1)
        s.synchronize()
        assert s.diagnostics()["nonfinite"] == 0
