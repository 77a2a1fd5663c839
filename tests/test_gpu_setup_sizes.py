"""Setup on the GPU at the mesh size where its scratch becomes one block, and
with tiles of every degree and general rows among them: the handle is the one
the host path builds (maps, tiles' numbers, phases) and its GatherScatter the
oracle's."""
import numpy as np
import pytest
import torch

from dawgs_gb300 import mesh, ogs
from helpers import random_ids, same_bits, signed_ids, values

pytestmark = pytest.mark.gpu


def check(ids, kind, oracle_mod):
    if kind == "signed":
        ids = signed_ids(ids, seed=17)
    k = ogs.Signed if kind == "signed" else ogs.Unsigned
    gd = ogs.ogs_t().Setup(ids.size, ids.copy(), None, k, ogs.Auto, False, maps="device")
    gh = ogs.ogs_t().Setup(ids.size, ids.copy(), None, k, ogs.Auto, False, maps="host")
    for x, y in zip(gd.maps(), gh.maps()):
        assert np.array_equal(x, y)
    assert gd.layout_stats() == gh.layout_stats()
    v = values(ids.size, np.float64, "add", seed=18)
    d = torch.from_numpy(v.copy()).cuda()
    gd.GatherScatter(d, 1, ogs.Add, ogs.Sym)
    torch.cuda.synchronize()
    assert same_bits(d.cpu().numpy(), oracle_mod.OracleOgs(ids.copy(), kind).gather_scatter(v.copy(), 1, "add", "sym"))
    return gd


@pytest.mark.parametrize("n", [32767, 32768])
@pytest.mark.parametrize("kind", ["unsigned", "signed"])
def test_scratch_in_pieces_and_in_one_block(cuda, oracle_mod, n, kind):
    check(random_ids(n, n // 3, seed=n), kind, oracle_mod)
