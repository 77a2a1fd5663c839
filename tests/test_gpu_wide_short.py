"""Rows above degree 8 at the edges of the wide tiles' batches of 12 and 24 members
and of the padding past which a handle has no wide tiles, against the oracle, bit
for bit: every pattern of Signed handles whose positive member is not the first."""
import numpy as np
import pytest
import torch

from dawgs_gb300 import mesh, ogs
from helpers import first_diff, same_bits, values

pytestmark = pytest.mark.gpu

TRANS = {"sym": ogs.Sym, "notrans": ogs.NoTrans, "trans": ogs.Trans}

# (degree, rows) ...: about 12 members on average (12, then 13 and more), rows longer than a batch among
# short ones, and one row of d members in a tile of 32 whose padding 32 d ids are around 2 (31 * 9 + d) + 2048
LISTS = [[(12, 40)], [(12, 39), (13, 1)], [(13, 40)], [(9, 60), (24, 1), (25, 1), (40, 1)], [(9, 33), (36, 3)],
         [(9, 31), (86, 1)], [(9, 31), (87, 1)], [(9, 31), (88, 1)], [(23, 5), (24, 70), (25, 5)]]


def one_positive(lists, seed):
    ids = np.concatenate([np.repeat(np.arange(n, dtype=np.int64) + 1 + 10000 * j, d)
                          for j, (d, n) in enumerate(lists)])
    ids = ids[np.argsort(mesh.uniform_values(ids.size, np.float64, 0.0, 1.0, seed), kind="stable")]
    pick = np.argsort(mesh.uniform_values(ids.size, np.float64, 0.0, 1.0, seed + 5), kind="stable")
    out = -ids
    _, at = np.unique(ids[pick], return_index=True)
    out[pick[at]] = ids[pick[at]]
    return out


@pytest.mark.parametrize("case", range(len(LISTS)))
def test_batches_and_padding(cuda, oracle_mod, case):
    ids = one_positive(LISTS[case], seed=case)
    ref = oracle_mod.OracleOgs(ids.copy(), "signed")
    for maps in ("host", "device"):
        g = ogs.ogs_t().Setup(ids.size, ids.copy(), None, ogs.Signed, maps=maps)
        for dtype in (np.float64, np.float32):
            for k in (1, 3):
                v = values(k * ids.size, dtype, "add", seed=k)
                for tname, trans in TRANS.items():
                    d = torch.from_numpy(v.copy()).cuda()
                    g.GatherScatter(d, k, ogs.Add, trans)
                    want = ref.gather_scatter(v.copy(), k, "add", tname)
                    assert same_bits(d.cpu().numpy(), want), (maps, k, tname, first_diff(d.cpu().numpy(), want))
                    if tname == "sym":
                        continue
                    gw = ref.gather(np.zeros(k * g.Ngather, dtype), v.copy(), k, "add", tname)
                    gv = torch.zeros(gw.size, dtype=d.dtype, device="cuda")
                    g.Gather(gv, torch.from_numpy(v.copy()).cuda(), k, ogs.Add, trans)
                    assert same_bits(gv.cpu().numpy(), gw), (maps, k, tname)
                    d = torch.from_numpy(v.copy()).cuda()
                    g.Scatter(d, gv, k, trans)
                    assert same_bits(d.cpu().numpy(), ref.scatter(v.copy(), gw, k, tname)), (maps, k, tname)
