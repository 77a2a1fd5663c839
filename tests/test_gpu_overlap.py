"""Calls whose kernels start before the work ahead of them has ended
(FieldArgs::overlap): long chains of library calls and torch kernels on one
stream, across two streams joined by events, and captured, against the same
arithmetic by torch on whole numbers."""
import numpy as np
import pytest
import torch

from dawgs_gb300 import mesh, ogs

pytestmark = pytest.mark.gpu


class Rows:
    """The handle's rows, by torch: GatherScatter, Gather and Scatter of int64 Add."""

    def __init__(self, ids, k):
        _, first, inv = np.unique(ids, return_index=True, return_inverse=True)
        rank = np.empty(first.size, np.int64)
        rank[np.argsort(first)] = np.arange(first.size)
        self.row = torch.from_numpy(rank[inv.reshape(-1)]).cuda()
        self.rows, self.k = first.size, k

    def gather(self, v):
        out = torch.zeros((self.rows, self.k), dtype=v.dtype, device="cuda")
        return out.index_add_(0, self.row, v.view(-1, self.k)).view(-1)

    def scatter(self, gv):
        return gv.view(-1, self.k)[self.row].reshape(-1).clone()


def handle(sizes):
    ids = mesh.box_ids(*sizes)
    return ids, ogs.ogs_t().Setup(ids.size, ids.copy(), None, ogs.Signed, ogs.Auto, True)


def chain(g, ref, q, gv, k, steps):
    """The library's calls and torch's on q and gv; with `ref`, by torch alone."""
    for s in range(steps):
        if ref is None:
            g.GatherScatter(q, k, ogs.Add, ogs.Sym)
            g.GatherScatter(q, k, ogs.Add, ogs.Sym)
            g.Gather(gv, q, k, ogs.Add, ogs.Trans)
            g.Scatter(q, gv, k, ogs.NoTrans)
        else:
            q.copy_(ref.scatter(ref.gather(q)))
            q.copy_(ref.scatter(ref.gather(q)))
            gv.copy_(ref.gather(q))
            q.copy_(ref.scatter(gv))
        if s % 3 == 0:
            q.remainder_(1000003).add_(s)
        elif s % 3 == 1:
            q.remainder_(65537)
            gv.add_(1)


@pytest.mark.parametrize("sizes,k", [((3, 3, 2, 2), 1), ((10, 10, 10, 3), 1), ((9, 8, 7, 5), 3), ((24, 24, 24, 7), 1)])
def test_chains(cuda, sizes, k):
    ids, g = handle(sizes)
    ref = Rows(ids, k)
    v = torch.from_numpy(mesh.uniform_values(k * ids.size, np.int64, -1000, 1000, 3)).cuda()
    want, wgv = v.clone(), torch.zeros(k * g.Ngather, dtype=torch.int64, device="cuda")
    chain(g, ref, want, wgv, k, 12)
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            q, gv = v.clone(), torch.zeros_like(wgv)
            chain(g, None, q, gv, k, 12)
        torch.cuda.synchronize()
        assert torch.equal(q, want) and torch.equal(gv, wgv)


@pytest.mark.parametrize("n,k", [(2000, 1), (60000, 1), (60000, 3), (900000, 1)])
def test_chains_with_general_rows(cuda, n, k):
    """Two launches a call: about half the nodes in rows of degree 20."""
    ids = mesh.uniform_values(n, np.int64, 1, 1 + n // 40, 6)
    few = mesh.uniform_values(n, np.int64, 0, 2, 7) == 0
    ids[few] = n + mesh.uniform_values(int(few.sum()), np.int64, 1, 1 + n // 4, 8)
    g = ogs.ogs_t().Setup(ids.size, ids.copy(), None, ogs.Signed, ogs.Auto, True)
    assert g.max_degree > 8
    ref = Rows(ids, k)
    v = torch.from_numpy(mesh.uniform_values(k * n, np.int64, -1000, 1000, 9)).cuda()
    want, wgv = v.clone(), torch.zeros(k * g.Ngather, dtype=torch.int64, device="cuda")
    chain(g, ref, want, wgv, k, 12)
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream()):
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            q, gv = v.clone(), torch.zeros_like(wgv)
            chain(g, None, q, gv, k, 12)
        torch.cuda.synchronize()
        assert torch.equal(q, want) and torch.equal(gv, wgv)


def test_two_streams(cuda):
    """A field handed back and forth between two streams by events, each with work of its own queued."""
    ids, g = handle((12, 11, 10, 4))
    ref = Rows(ids, 1)
    v = torch.from_numpy(mesh.uniform_values(ids.size, np.int64, -1000, 1000, 4)).cuda()
    want = v.clone()
    for _ in range(20):
        want = ref.scatter(ref.gather(want)).remainder_(7919)
    streams, other = [torch.cuda.Stream(), torch.cuda.Stream()], torch.ones(1 << 22, device="cuda")
    q = v.clone()
    torch.cuda.synchronize()
    e = None
    for s in range(20):
        with torch.cuda.stream(streams[s % 2]):
            other.mul_(1.0)
            if e is not None:
                streams[s % 2].wait_event(e)
            g.GatherScatter(q, 1, ogs.Add, ogs.Sym)
            q.remainder_(7919)
            e = torch.cuda.Event()
            e.record()
            g.GatherScatter(v, 1, ogs.Max, ogs.Sym)
    torch.cuda.synchronize()
    assert torch.equal(q, want)


def test_captured(cuda):
    ids, g = handle((10, 10, 10, 3))
    ref = Rows(ids, 1)
    v = torch.from_numpy(mesh.uniform_values(ids.size, np.int64, -1000, 1000, 5)).cuda()
    want, wgv = v.clone(), torch.zeros(g.Ngather, dtype=torch.int64, device="cuda")
    chain(g, ref, want, wgv, 1, 6)
    q, gv = v.clone(), torch.zeros_like(wgv)
    g.GatherScatter(q, 1, ogs.Add, ogs.Sym)  # not captured: modules load
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(g, None, q, gv, 1, 6)
    for _ in range(3):
        q.copy_(v)
        gv.zero_()
        graph.replay()
        g.GatherScatter(v.clone(), 1, ogs.Add, ogs.Sym)
        torch.cuda.synchronize()
        assert torch.equal(q, want) and torch.equal(gv, wgv)
