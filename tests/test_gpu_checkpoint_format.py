"""The bytes of a checkpoint do not change from build to build of one format version:
psi and theta as long as the handle's cells (rows padded to 8, domains to 32), with
nothing after the last domain's.  A checkpoint whose two arrays are rounded up to 32
cells, as some builds wrote it, restores too."""
import struct

import numpy as np
import pytest

import dhara_b200 as db
from dhara_b200 import inputs

pytestmark = pytest.mark.gpu

HEADER = 8 + 2 * 4 + 2 * 8 + 2 * 4  # magic; version, domains; cells, columns; record sizes


def fresh(shapes):
    doms = [inputs.make_domain(*n, seed=i, rain_mm_per_h=30.0, nsteps=4, precision=db.MIXED, krylov_tol=1e-10)
            for i, n in enumerate(shapes)]
    s = db.Solver([d.params for d in doms])
    for i, d in enumerate(doms):
        s.load(d, i)
    s.prepare()
    return s


@pytest.mark.parametrize("shapes", [[(9, 37, 7)], [(5, 3, 1)], [(24, 20, 10), (9, 37, 7)], [(16, 8, 4)]])
def test_checkpoint_layout(gpu, shapes):
    cells = 0
    for nx, ny, nz in shapes:
        cells = (cells + 31) // 32 * 32 + (nx + 7) // 8 * 8 * ny * nz
    slab, cols, nd = (cells + 31) // 32 * 32, sum(nx * ny for nx, ny, _ in shapes), len(shapes)
    with fresh(shapes) as s:
        s.step(2)
        ck = s.checkpoint()
        want = [s.download("psi", i) for i in range(nd)], [s.download("theta", i) for i in range(nd)]
        pctrl, diag = struct.unpack_from("<2i", ck, HEADER - 8)
    assert struct.unpack_from("<2q", ck, 16) == (cells, cols)
    assert ck.size == HEADER + 12 * nd + 8 * (2 * cells + 4 * cols) + nd * (pctrl + diag + 16)
    # the same with both arrays rounded up
    o = HEADER + 12 * nd
    pad = np.full(8 * (slab - cells), 255, np.uint8)  # NaN: must not be read
    wide = np.concatenate([ck[:o], ck[o:o + 8 * cells], pad, ck[o + 8 * cells:o + 16 * cells], pad, ck[o + 16 * cells:]])
    struct.pack_into("<q", wide, 16, slab)
    for buf in (ck, wide):
        with fresh(shapes) as s:
            s.step(1)
            s.restore(buf)
            again = s.checkpoint()
            got = [s.download("psi", i) for i in range(nd)], [s.download("theta", i) for i in range(nd)]
        assert np.array_equal(again, ck)
        for a, b in zip(want[0] + want[1], got[0] + got[1]):
            assert np.array_equal(a, b)
