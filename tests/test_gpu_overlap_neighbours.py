"""What a kernel of another library that is launched with programmatic stream
serialization behind a call finds before its own wait: all work ahead of the call
done; and, behind a handle without overlap or a captured call, the call too."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import torch

from dawgs_gb300 import build, mesh, ogs

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(cuda, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("probe") / "overlap_probe.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-cudart", "static",
                    os.path.join(HERE, "cpp", "overlap_probe.cu"), "-o", so], check=True, capture_output=True)
    P = C.CDLL(so)
    P.probe_ahead.argtypes = [C.c_void_p, C.c_longlong, C.c_void_p]
    P.probe_behind.argtypes = [C.c_void_p] * 4
    return P


def seen_behind(probe, g, call, captured=False):
    """(ahead done, first value before the wait, after it) with the field at 1 before the call."""
    q = torch.ones(g.N, dtype=torch.float64, device="cuda")
    x = torch.full((g.Ngather,), 7.0, dtype=torch.float64, device="cuda")
    out = x if call == "gather" else q
    calls = {"gather_scatter": lambda: g.GatherScatter(q, 1, ogs.Add, ogs.Sym),
             "gather": lambda: g.Gather(x, q, 1, ogs.Add, ogs.Trans),
             "scatter": lambda: g.Scatter(q, x, 1, ogs.NoTrans)}
    calls[call]()  # modules load
    q.fill_(1.0)
    if call != "scatter":
        x.fill_(0.0)
    done = torch.zeros(1, dtype=torch.int32, device="cuda")
    seen = torch.zeros(3, dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        def all_three():
            s = torch.cuda.current_stream().cuda_stream
            assert probe.probe_ahead(done.data_ptr(), 400000, s) == 0
            calls[call]()
            assert probe.probe_behind(done.data_ptr(), out.data_ptr(), seen.data_ptr(), s) == 0
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                all_three()
            graph.replay()
        else:
            all_three()
    torch.cuda.synchronize()
    return seen.cpu().tolist()


@pytest.mark.parametrize("call", ["gather_scatter", "gather", "scatter"])
@pytest.mark.parametrize("side,p", [(4, 3), (12, 5)])
def test_work_ahead_of_the_call_is_done(probe, side, p, call):
    ids = mesh.box_ids(side, side, side, p)
    order = np.argsort(-ids, kind="stable")  # first value in a row of several members
    ids = np.ascontiguousarray(ids[order][::-1])
    ids[0] = ids[-1] = ids.max() + 1
    want = 7.0 if call == "scatter" else 2.0
    for overlap in (True, False):
        g = ogs.ogs_t().Setup(ids.size, ids.copy(), None, ogs.Signed, ogs.Auto, True, overlap=overlap)
        for captured in (False, True):
            for _ in range(3):
                seen = seen_behind(probe, g, call, captured)
                assert seen[0] == 1 and seen[2] == want, (overlap, captured, seen)
                if captured or not overlap:
                    assert seen[1] == want, (overlap, captured, seen)
