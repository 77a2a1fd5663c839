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


def degrees_ids(n, seed):
    """n nodes in groups of degree 1 to 40, most of them small, in random order."""
    d = mesh.uniform_values(n, np.int64, 1, 11, seed)
    d = np.where(d == 10, mesh.uniform_values(n, np.int64, 9, 41, seed + 1), d)
    ids = np.repeat(np.arange(1, n + 1), d)[:n]
    return ids[np.argsort(mesh.uniform_values(n, np.float64, 0.0, 1.0, seed + 2), kind="stable")].astype(np.int64)


@pytest.mark.parametrize("n", [1, 33, 4001, 900000])
@pytest.mark.parametrize("kind", ["unsigned", "signed"])
def test_tiles_of_every_degree_in_row_order(cuda, oracle_mod, n, kind):
    """The tile lists: one tile of one row up to hundreds of tiles in every
    bucket, and general tiles between them."""
    g = check(degrees_ids(n, seed=n), kind, oracle_mod)
    s = g.layout_stats()
    if n >= 4001:
        assert len(s["rows_by_degree"]) == 8 and s["ngeneral_tiles"] >= 1
    if n == 900000:
        assert s["ngeneral_tiles"] > 1 and len(s["phases"]) > 1  # phases are cut along the list
