"""Steps with a high limit on Picard iterations in the launch-per-kernel schedule: small
handles queue launches for the first 32 iterations and one launch for the rest
(separate_iterations, csrc/subsurface.cu), so a step that converges early does not pay
for the limit.  The same bits as the fused schedule, which ends its loop on the
device, for steps that stop before, at and after the 32nd iteration and for batches
whose domains do, with both solvers and with Dirichlet faces; and the launches."""
import numpy as np
import pytest

import dhara_b200 as db
from dhara_b200 import inputs

from test_gpu_dirichlet import domain_with_faces

pytestmark = pytest.mark.gpu

FIELDS = ("psi", "theta", "ponding", "waterelev")
COUNTS = ("picard_iters_total", "krylov_iters_total", "refine_iters_total", "picard_nonconverged",
          "krylov_nonconverged", "krylov_relres_last", "picard_err_last", "mb_subsurface_cum")


def domain(limit, tol, prec, shape=(24, 13, 6), seed=3):
    return inputs.make_domain(*shape, seed=seed, precision=prec, rain_mm_per_h=30.0, nsteps=3, krylov_tol=1e-10,
                              krylov_maxiter=2000, picard_rule=db.PICARD_PSI_ABSOLUTE, picard_tol=tol,
                              picard_maxiter=limit)


def run(doms, fused, nsteps=3, choose=None, graph=False):
    s = db.Solver([d.params for d in doms])
    for i, d in enumerate(doms):
        s.load(d, i)
    s.prepare()
    c = s.launch_config()
    s.set_launch_config(c["krylov_blocks_per_sm"], c["overland_resident"], c["overland_blocks_per_sm"],
                        fused_step=fused, krylov_solver=choose)
    n0 = s.launch_count()
    s.step(nsteps, graph=graph)
    s.synchronize()
    out = [({k: s.download(k, i) for k in FIELDS}, s.diagnostics(i)) for i in range(len(doms))]
    n = s.launch_count() - n0
    s.close()
    return out, n


def same(a, b):
    for (sa, da), (sb, dbg) in zip(a, b):
        for k in FIELDS:
            assert np.array_equal(sa[k], sb[k]), k
        for k in COUNTS:
            assert da[k] == dbg[k], k


@pytest.mark.parametrize("prec", [db.FP64, db.MIXED])
@pytest.mark.parametrize("limit", [32, 33, 45])
@pytest.mark.parametrize("tol", [1e-1, 1e-300])
def test_limit_gives_the_fused_steps_bits(gpu, limit, tol, prec):
    doms = [domain(limit, tol, prec)]
    for choose in (1, 2):
        (a, n), (b, _) = run(doms, 0, choose=choose), run(doms, 1, choose=choose)
        same(a, b)
        assert (a[0][1]["picard_iters_last"] == limit) == (tol == 1e-300)
        assert n <= 3 * (2 + 3 * 32 + 1 + 3)
    (g, _) = run(doms, 0, choose=2, graph=True)
    same(g, b)


@pytest.mark.parametrize("prec", [db.FP64, db.MIXED])
def test_batch_of_early_and_late_domains(gpu, prec):
    doms = [domain(12 + 6 * i, 1e-300 if i % 2 else 1e-1, prec, (20 + i, 9, 4 + i % 3), i) for i in range(7)]
    (a, _), (b, _) = run(doms, 0), run(doms, 1)
    same(a, b)
    assert [r[1]["picard_iters_last"] for r in a][1::2] == [18, 30, 42]


def test_with_dirichlet_faces(gpu):
    d = domain_with_faces({"west": 0.2, "bottom": -0.1})
    d.params.picard_maxiter = 40
    d.params.picard_tol = 1e-300
    (a, _), (b, _) = run([d], 0), run([d], 1)
    same(a, b)
    assert a[0][1]["picard_iters_last"] == 40
