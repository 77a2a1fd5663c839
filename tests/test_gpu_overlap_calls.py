"""Chains of calls on one stream whose kernels start before the work ahead has
ended, of the kinds that wait at their start (masked patterns, components) and of
separate arrays: the same bits as on a handle without overlap, one call at a time."""
import numpy as np
import pytest
import torch

from dawgs_gb300 import mesh, ogs
from helpers import values

pytestmark = pytest.mark.gpu


def one_positive(ids, seed):
    """Signed ids, one positive a group and not its first."""
    pick = np.argsort(mesh.uniform_values(ids.size, np.float64, 0.0, 1.0, seed), kind="stable")
    out = -ids
    _, at = np.unique(ids[pick], return_index=True)
    out[pick[at]] = ids[pick[at]]
    return out


def chain(g, q, gv, many, k, wait):
    for s in range(8):
        calls = [lambda: g.GatherScatter(q, k, ogs.Max, ogs.Trans), lambda: g.GatherScatter(q, k, ogs.Add, ogs.NoTrans),
                 lambda: g.Gather(gv, q, k, ogs.Min, ogs.NoTrans), lambda: g.Scatter(q, gv, k, ogs.Trans),
                 lambda: g.GatherScatter(q, k, ogs.Max, ogs.Sym), lambda: g.GatherScatterMany(many, ogs.Add, ogs.Sym),
                 lambda: g.GatherScatterMany(many, ogs.Max, ogs.Trans), lambda: g.Gather(gv, q, k, ogs.Add, ogs.Trans),
                 lambda: q.remainder_(1000003).add_(s), lambda: [m.remainder_(65537) for m in many]]
        for call in calls:
            call()
            if wait:
                torch.cuda.synchronize()


@pytest.mark.parametrize("k", [1, 3])
@pytest.mark.parametrize("sizes", [(3, 3, 2, 2), (10, 10, 10, 3), (9, 8, 7, 5), (20, 20, 20, 7)])
def test_chains(cuda, sizes, k):
    ids = one_positive(mesh.box_ids(*sizes), seed=5)
    v = torch.from_numpy(values(k * ids.size, np.int64, "add", seed=6)).cuda()
    vs = torch.from_numpy(values(3 * ids.size, np.int64, "add", seed=7)).cuda()
    got = []
    for overlap in (False, True, True):
        g = ogs.ogs_t().Setup(ids.size, ids.copy(), None, ogs.Signed, overlap=overlap)
        assert g.gather_defined
        with torch.cuda.stream(torch.cuda.Stream()):
            q, m = v.clone(), vs.clone()
            gv = torch.zeros(k * g.Ngather, dtype=torch.int64, device="cuda")
            chain(g, q, gv, list(m.view(3, -1).unbind(0)), k, wait=not overlap)
        torch.cuda.synchronize()
        got.append((q, gv, m))
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))
