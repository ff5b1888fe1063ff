"""The sharded ensemble (dhara_b200.ensemble.run_sharded) with other numbers of ranks:
each rank's share run here one after the other, the gather left out (its host side is
tested on gloo in test_dist.py).  A domain's diagnostics are the same bits whichever
domains it shares a handle with: 256 domains in one handle are many tiles per SM, a
share of 32 few, where a handle by itself would choose the other 3D solver."""
import pytest

from dhara_b200 import ensemble as ens
from dhara_b200 import inputs

pytestmark = pytest.mark.gpu


def test_any_number_of_ranks_gives_the_same_bits(gpu, monkeypatch):
    monkeypatch.setattr(ens, "gather_diagnostics", lambda local, world: dict(local))
    doms = inputs.ensemble(256, nsteps=2)
    _, _, whole = ens.run_sharded(doms, 2, 0, 1)
    seen = set()
    for world, ranks in ((2, (0, 1)), (8, (0, 3, 7)), (64, (5,))):
        for rank in ranks:
            _, _, part = ens.run_sharded(doms, 2, rank, world)
            for i, dg in part.items():
                seen.add(i)
                for k in dg:
                    if k != "launch_config":
                        assert dg[k] == whole[i][k], (world, i, k)
                assert dg["launch_config"]["krylov_solver"] == whole[i]["launch_config"]["krylov_solver"] == 2
    assert len(seen) == 256
