"""Scatter in node order where its CTAs become larger (ogs_scatter.cuh), against
the oracle, bit for bit."""
import numpy as np
import pytest
import torch

from dawgs_gb300 import mesh, ogs
from helpers import first_diff, random_ids, same_bits, values

pytestmark = pytest.mark.gpu


def scattered(oracle_mod, ids, k, dtype):
    ref = oracle_mod.OracleOgs(ids.copy(), "signed", unique=True)
    g = ogs.ogs_t().Setup(ids.size, ids.copy(), None, ogs.Signed, ogs.Auto, True)
    gv = values(k * g.Ngather, dtype, "add", seed=k)
    v0 = values(k * ids.size, dtype, "add", seed=k + 1)
    for tname, trans in (("notrans", ogs.NoTrans), ("trans", ogs.Trans)):
        v = torch.from_numpy(v0.copy()).cuda()
        g.Scatter(v, torch.from_numpy(gv).cuda(), k, trans)
        got, want = v.cpu().numpy(), ref.scatter(v0.copy(), gv, k, tname)
        assert same_bits(got, want), (tname, first_diff(got, want))


# 512 CTAs of 8 warps: words of 32 nodes, 8, 4, 2 and 1 a warp
@pytest.mark.parametrize("k,words", [(1, 64), (2, 32), (3, 16), (5, 8), (8, 8)])
@pytest.mark.parametrize("more", [-31, 0, 1, 33])
def test_at_the_larger_ctas(cuda, oracle_mod, k, words, more):
    n = 511 * words * 32 + more
    for dtype in (np.float64, np.float32):
        scattered(oracle_mod, random_ids(n, n // 3, seed=n, zero_frac=0.1), k, dtype)


@pytest.mark.parametrize("k", [7, 8, 9, 13, 15, 16, 17])
@pytest.mark.parametrize("n", [33, 4097, 140001])
def test_components_up_to_the_tiles(cuda, oracle_mod, n, k):
    """Each count of components is a kernel of its own up to 64 bytes a node."""
    ids = random_ids(n, n // 3, seed=n + k, zero_frac=0.05)
    for dtype in (np.float32, np.int32, np.float64, np.int64):
        scattered(oracle_mod, ids, k, dtype)


@pytest.mark.parametrize("k", [1, 3, 9])
@pytest.mark.parametrize("zeros", [0.22, 0.28, 0.99])
def test_where_few_nodes_take_part(cuda, oracle_mod, zeros, k):
    """Both sides of the share of nodes from which a Scatter runs in node order."""
    n = 70001
    ids = random_ids(n, n // 3, seed=k, zero_frac=zeros)
    scattered(oracle_mod, ids, k, np.float64)
