"""Degree-1 rows as lone tiles (the ltiles of ogs_async.cuh) against the oracle,
bit for bit: node counts around a tile of 256 and its 16-byte vectors, meshes of
mostly lone nodes with shared rows among them, zero ids, the values that the
fold from the identity changes, fields off the 16-byte boundary, separate
arrays, Signed handles, both builds of the maps."""
import numpy as np
import pytest
import torch

from dawgs_gb300 import mesh, ogs
from helpers import first_diff, same_bits, signed_ids, values

pytestmark = pytest.mark.gpu

SPECIAL = {np.float64: [-0.0, 0.0, np.inf, -np.inf, np.finfo(np.float64).max, -np.finfo(np.float64).max, 5e-324],
           np.float32: [-0.0, 0.0, np.inf, -np.inf, np.finfo(np.float32).max, -np.finfo(np.float32).max, 1e-45],
           np.int64: [0, -2**63, -2**63 + 1, 2**63 - 1], np.int32: [0, -2**31, -2**31 + 1, 2**31 - 1]}


def mostly_lone(n, seed):
    """About two thirds lone nodes, the others in rows of two to four, some zeros."""
    ids = np.arange(n, dtype=np.int64) + 1
    r = mesh.uniform_values(n, np.int64, 0, 9, seed)
    shared = np.nonzero(r < 3)[0]
    ids[shared] = n + 1 + mesh.uniform_values(shared.size, np.int64, 0, max(1, shared.size // 3), seed + 1)
    ids[mesh.uniform_values(n, np.int64, 0, 40, seed + 2) == 0] = 0
    return ids


def field(n, dtype, op, seed):
    v = values(n, dtype, op, seed)
    at = mesh.uniform_values(n, np.int64, 0, 5, seed + 7) == 0
    s = np.array(SPECIAL[dtype], dtype)
    v[at] = s[mesh.uniform_values(n, np.int64, 0, s.size, seed + 8)][at]
    return v


@pytest.mark.parametrize("dtype", list(SPECIAL))
@pytest.mark.parametrize("n", [2, 255, 256, 257, 511, 515, 1030, 70003])
def test_lone(cuda, oracle_mod, n, dtype):
    base = mostly_lone(n, seed=n)
    if not base.any():
        base[0] = 1
    for kind, maps in (("unsigned", "host"), ("unsigned", "device"), ("unique", "device")):
        g = ogs.ogs_t().Setup(n, base.copy(), None, ogs.Unsigned if kind == "unsigned" else ogs.Signed, ogs.Auto,
                              kind == "unique", maps=maps)
        ref = oracle_mod.OracleOgs(base.copy(), kind if kind == "unsigned" else "signed", unique=kind == "unique")
        for op in ("add", "mul", "max", "min"):
            v = field(n, dtype, op, seed=n)
            with np.errstate(all="ignore"):
                want = ref.gather_scatter(v.copy(), 1, op, "sym")
            room = torch.zeros(n + 1, dtype=torch.from_numpy(v).dtype, device="cuda")
            for at in (0, 1):  # on and off the boundary
                d = room[at:at + n]
                d.copy_(torch.from_numpy(v))
                g.GatherScatter(d, 1, ogs.Op[op.capitalize()], ogs.Sym)
                got = d.cpu().numpy()
                ok = ~(np.isnan(got) & np.isnan(want)) if got.dtype.kind == "f" else np.ones(n, bool)
                assert same_bits(got[ok], want[ok]), (kind, op, at, first_diff(got, want))
            vs = [values(n, dtype, op, seed=j) for j in range(3)]
            ds = [torch.from_numpy(x.copy()).cuda() for x in vs]
            g.GatherScatterMany(ds, ogs.Op[op.capitalize()], ogs.Sym)
            for x, d in zip(vs, ds):
                assert same_bits(d.cpu().numpy(), ref.gather_scatter(x.copy(), 1, op, "sym")), (kind, op)


@pytest.mark.parametrize("dtype", list(SPECIAL))
@pytest.mark.parametrize("n", [2, 255, 256, 257, 515, 4100, 70003])
def test_lone_gathered(cuda, oracle_mod, n, dtype):
    """Gather on Signed unique handles: a lone node's row follows from its word's first members."""
    base = mostly_lone(n, seed=n + 1)
    if not base.any():
        base[0] = 1
    ref = oracle_mod.OracleOgs(base.copy(), "signed", unique=True)
    for maps in ("host", "device"):
        g = ogs.ogs_t().Setup(n, base.copy(), None, ogs.Signed, ogs.Auto, True, maps=maps)
        for op in ("add", "mul", "max", "min"):
            for tname, trans in (("trans", ogs.Trans), ("notrans", ogs.NoTrans)):
                v = field(n, dtype, op, seed=n)
                want = np.zeros(ref.Ngather, dtype)
                with np.errstate(all="ignore"):
                    ref.gather(want, v, 1, op, tname)
                gv = torch.zeros(want.size, dtype=torch.from_numpy(v).dtype, device="cuda")
                g.Gather(gv, torch.from_numpy(v.copy()).cuda(), 1, ogs.Op[op.capitalize()], trans)
                got = gv.cpu().numpy()
                ok = ~(np.isnan(got) & np.isnan(want)) if got.dtype.kind == "f" else np.ones(want.size, bool)
                assert same_bits(got[ok], want[ok]), (maps, op, tname, first_diff(got, want))


def test_signed_patterns_and_host_buffers(cuda, oracle_mod):
    """Handles with lone tiles keep the other tiles for masked patterns and host buffers."""
    ids = signed_ids(mostly_lone(70003, seed=1), seed=4)
    g = ogs.ogs_t().Setup(ids.size, ids.copy(), None, ogs.Signed)
    ref = oracle_mod.OracleOgs(ids.copy(), "signed")
    v = values(ids.size, np.float64, "add", seed=2)
    for tname, trans in (("sym", ogs.Sym), ("notrans", ogs.NoTrans), ("trans", ogs.Trans)):
        want = ref.gather_scatter(v.copy(), 1, "add", tname)
        d = torch.from_numpy(v.copy()).cuda()
        g.GatherScatter(d, 1, ogs.Add, trans)
        h = torch.from_numpy(v.copy()).pin_memory()
        g.GatherScatter(h, 1, ogs.Add, trans)
        assert same_bits(d.cpu().numpy(), want) and same_bits(h.numpy(), want), tname
