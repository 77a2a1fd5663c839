"""Scatter in node order (ogs_scatter.cuh) against the oracle, bit for bit, at
the edges of its words (32 nodes), items (up to 256 nodes a warp) and component
runs, with zero ids, on handles whose positive member is not the first, built
on either side."""
import numpy as np
import pytest
import torch

from dawgs_gb300 import mesh, ogs
from helpers import first_diff, random_ids, same_bits, values

pytestmark = pytest.mark.gpu

_TORCH = {np.float32: torch.float32, np.float64: torch.float64, np.int32: torch.int32, np.int64: torch.int64}
TRANS = {"notrans": ogs.NoTrans, "trans": ogs.Trans}


def one_positive(n, seed):
    """Ids with zeros where each group's positive member is a drawn one."""
    ids = random_ids(n, max(1, n // 3), seed, zero_frac=0.1)
    pick = np.argsort(mesh.uniform_values(n, np.float64, 0.0, 1.0, seed + 5), kind="stable")
    out = -ids
    _, at = np.unique(ids[pick], return_index=True)
    out[pick[at]] = ids[pick[at]]
    return out


@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.int64, np.int32])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 9, 33])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 257, 2049])
def test_scatter(cuda, oracle_mod, n, k, dtype):
    ids = one_positive(n, seed=n + k)
    if not ids.any():
        ids[0] = 1
    ref = oracle_mod.OracleOgs(ids.copy(), "signed")
    for maps in ("host", "device"):
        g = ogs.ogs_t().Setup(n, ids.copy(), None, ogs.Signed, maps=maps)
        assert g.gather_defined
        for tname, trans in TRANS.items():
            gv = values(k * g.Ngather, dtype, "add", seed=k)
            v0 = values(k * n, dtype, "add", seed=k + 1)
            v = torch.from_numpy(v0.copy()).cuda()
            g.Scatter(v, torch.from_numpy(gv).cuda(), k, trans)
            torch.cuda.synchronize()
            got, want = v.cpu().numpy(), ref.scatter(v0.copy(), gv, k, tname)
            assert same_bits(got, want), (maps, tname, first_diff(got, want))
