"""Rows above degree 8 as wide tiles (ogs_wide.cuh) against the oracle, bit for
bit: degrees around the batches in flight, row counts around a tile and around
the number of tiles that go along with the exact-degree rows, every layout of
the components, N masks, and a row so long that the handle keeps CTA tiles."""
import numpy as np
import pytest
import torch

from dawgs_gb300 import mesh, ogs
from helpers import first_diff, same_bits, signed_ids, values

pytestmark = pytest.mark.gpu

TRANS = {"sym": ogs.Sym, "notrans": ogs.NoTrans, "trans": ogs.Trans}

# (degree, rows): one row, a tile less one, a tile, one more; 130 tiles of degree 9; mixed
LISTS = [[(9, 1)], [(23, 31), (2, 5)], [(24, 32), (1, 3)], [(25, 33)], [(9, 4160), (3, 40)],
         [(8, 10), (16, 20), (17, 20), (48, 13), (64, 3)], [(10, 40), (5000, 1)]]


def ids_of(lists, seed):
    ids = np.concatenate([np.repeat(np.arange(n, dtype=np.int64) + 1 + 10000 * j, d)
                          for j, (d, n) in enumerate(lists)])
    order = np.argsort(mesh.uniform_values(ids.size, np.float64, 0.0, 1.0, seed), kind="stable")
    return ids[order]


@pytest.mark.parametrize("dtype,op", [(np.float64, "add"), (np.float32, "mul"), (np.int64, "max"), (np.int32, "add")])
@pytest.mark.parametrize("case", range(len(LISTS)))
def test_wide_rows(cuda, oracle_mod, case, dtype, op):
    base = ids_of(LISTS[case], seed=case)
    for kind, maps in (("unsigned", "device"), ("signed", "host"), ("signed", "device")):
        ids = signed_ids(base, seed=case + 3) if kind == "signed" else base.copy()
        g = ogs.ogs_t().Setup(ids.size, ids.copy(), None, ogs.Signed if kind == "signed" else ogs.Unsigned, maps=maps)
        ref = oracle_mod.OracleOgs(ids.copy(), kind)
        for k in (1, 3):
            for tname, trans in TRANS.items():
                v = values(k * ids.size, dtype, op, seed=k)
                want = ref.gather_scatter(v.copy(), k, op, tname)
                d = torch.from_numpy(v.copy()).cuda()
                g.GatherScatter(d, k, ogs.Op[op.capitalize()], trans)
                assert same_bits(d.cpu().numpy(), want), (kind, k, tname, first_diff(d.cpu().numpy(), want))
        vs = [values(ids.size, dtype, op, seed=j) for j in range(2)]
        ds = [torch.from_numpy(x.copy()).cuda() for x in vs]
        g.GatherScatterMany(ds, ogs.Op[op.capitalize()], ogs.Sym)
        for x, d in zip(vs, ds):
            assert same_bits(d.cpu().numpy(), ref.gather_scatter(x.copy(), 1, op, "sym")), kind


@pytest.mark.parametrize("case", range(len(LISTS)))
def test_wide_rows_gathered(cuda, oracle_mod, case):
    """Gather on the Signed unique handle, Gather and Scatter of an operator over the same maps."""
    ids = ids_of(LISTS[case], seed=case)
    ref = oracle_mod.OracleOgs(ids.copy(), "signed", unique=True)
    g = ogs.ogs_t().Setup(ids.size, ids.copy(), None, ogs.Signed, ogs.Auto, True)
    op = ogs.ogs_t().SetupMaps(ids.size, *g.maps()[:2])
    for k in (1, 2):
        v = values(k * ids.size, np.float64, "add", seed=k)
        gw = np.zeros(k * ref.Ngather)
        ref.gather(gw, v, k, "add", "trans")
        for h in (g, op):
            gv = torch.zeros(gw.size, dtype=torch.float64, device="cuda")
            h.Gather(gv, torch.from_numpy(v.copy()).cuda(), k, ogs.Add, ogs.Trans)
            assert same_bits(gv.cpu().numpy(), gw)
            d = torch.from_numpy(v.copy()).cuda()
            h.Scatter(d, gv, k, ogs.NoTrans)
            assert same_bits(d.cpu().numpy(), ref.scatter(v.copy(), gw, k, "notrans"))
