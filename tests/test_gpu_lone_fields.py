"""Lone tiles (ogs_async.cuh, ogs_warp.cuh) where the rules take them and where
they must not be taken, against the oracle, bit for bit: NaN and infinities, Gather
of fields large enough, and on handles that have lone tiles the masked patterns and
page-locked host fields, which keep the ordinary tiles."""
import numpy as np
import pytest
import torch

from dawgs_gb300 import mesh, ogs
from helpers import first_diff, same_bits, values
from test_gpu_lone_tiles import field, mostly_lone

pytestmark = pytest.mark.gpu


def lone_handle(n, kind, seed, oracle_mod):
    ids = mostly_lone(n, seed)
    g = ogs.ogs_t().Setup(n, ids.copy(), None, ogs.Signed if kind == "signed" else ogs.Unsigned, ogs.Auto,
                          kind == "signed")
    # 65 % of the nodes and every row with a positive member: what gets, and always takes, lone tiles
    assert g.layout_stats()["rows_by_degree"][1] * 20 >= n * 13 and g.NlocalP == g.NlocalT
    return g, oracle_mod.OracleOgs(ids.copy(), kind, unique=kind == "signed")


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [257, 4100, 70003])
def test_nan(cuda, oracle_mod, n, dtype):
    """NaN of either sign, quiet as the GPU makes it and with other bits: Max and Min turn a lone one
    into the identity, Add leaves a NaN (whose bits a fold may change, so only its being one is compared)."""
    g, ref = lone_handle(n, "unsigned", n, oracle_mod)
    v = field(n, dtype, "add", seed=n)
    nan = np.array([np.nan, -np.nan, np.nan], dtype)
    nan[2:].view(np.uint64 if dtype == np.float64 else np.uint32)[:] |= 5
    at = mesh.uniform_values(n, np.int64, 0, 4, n + 1) == 0
    v[at] = nan[mesh.uniform_values(n, np.int64, 0, 3, n + 2)][at]
    for op in ("max", "min", "add"):
        with np.errstate(all="ignore"):
            want = ref.gather_scatter(v.copy(), 1, op, "sym")
        d = torch.from_numpy(v.copy()).cuda()
        g.GatherScatter(d, 1, ogs.Op[op.capitalize()], ogs.Sym)
        got = d.cpu().numpy()
        if op == "add":
            assert np.array_equal(np.isnan(got), np.isnan(want))
            got, want = got[~np.isnan(got)], want[~np.isnan(want)]
        assert same_bits(got, want), (op, first_diff(got, want))


@pytest.mark.parametrize("dtype,n", [(np.float64, 3932160 + 33), (np.float32, 7864320 + 290), (np.int64, 3932160 + 1)])
def test_gather_of_a_large_field(cuda, oracle_mod, dtype, n):
    g, ref = lone_handle(n, "signed", n, oracle_mod)
    for op in ("add", "max"):
        v = field(n, dtype, op, seed=n)
        with np.errstate(all="ignore"):
            want = ref.gather(np.zeros(g.Ngather, dtype), v.copy(), 1, op, "trans")
        gv = torch.zeros(g.Ngather, dtype=torch.from_numpy(v).dtype, device="cuda")
        g.Gather(gv, torch.from_numpy(v.copy()).cuda(), 1, ogs.Op[op.capitalize()], ogs.Trans)
        got = gv.cpu().numpy()
        ok = ~(np.isnan(got) & np.isnan(want)) if got.dtype.kind == "f" else np.ones(got.size, bool)
        assert same_bits(got[ok], want[ok]), (op, first_diff(got, want))


@pytest.mark.parametrize("kind", ["signed", "unsigned"])
@pytest.mark.parametrize("n", [515, 300001])
def test_masked_patterns_and_host_fields(cuda, oracle_mod, n, kind):
    g, ref = lone_handle(n, kind, n + 7, oracle_mod)
    assert n < 100000 or len(g.layout_stats()["phases"]) > 1  # sliced
    for tname, trans in (("sym", ogs.Sym), ("notrans", ogs.NoTrans), ("trans", ogs.Trans)):
        for op in ("add", "max"):
            v = values(n, np.float64, op, seed=3)
            want = ref.gather_scatter(v.copy(), 1, op, tname)
            d = torch.from_numpy(v.copy()).cuda()
            g.GatherScatter(d, 1, ogs.Op[op.capitalize()], trans)
            assert same_bits(d.cpu().numpy(), want), (tname, op)
            h = torch.from_numpy(v.copy()).pin_memory()
            g.GatherScatter(h, 1, ogs.Op[op.capitalize()], trans)
            assert same_bits(h.numpy(), want), (tname, op, "host")
    if kind == "signed":
        v = values(n, np.float64, "add", seed=4)
        for tname, trans in (("notrans", ogs.NoTrans), ("trans", ogs.Trans)):
            want = ref.gather(np.zeros(g.Ngather), v.copy(), 1, "add", tname)
            gv = torch.zeros(g.Ngather, dtype=torch.float64).pin_memory()
            g.Gather(gv, torch.from_numpy(v.copy()).pin_memory(), 1, ogs.Add, trans)
            assert same_bits(gv.numpy(), want), tname
            h = torch.from_numpy(v.copy()).pin_memory()
            g.Scatter(h, gv, 1, trans)
            assert same_bits(h.numpy(), ref.scatter(v.copy(), want.copy(), 1, tname)), tname
