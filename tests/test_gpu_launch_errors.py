"""A launch that the runtime refuses on the host is that call's error and no other's."""
import ctypes as C
import os

import numpy as np
import pytest
import torch

from dawgs_gb300 import _lib, build, mesh, ogs
from helpers import same_bits, values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["scatter", "gather", "gather_scatter"])
def test_refused_launch_leaves_the_next_call_alone(cuda, oracle_mod, call):
    """Work on the legacy stream while a blocking stream is captured is refused."""
    rt = C.CDLL(os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "lib64", "libcudart.so"))
    ids = mesh.box_ids(6, 6, 6, 3)
    g = ogs.ogs_t().Setup(ids.size, ids.copy(), None, ogs.Signed, ogs.Auto, True)
    v = values(ids.size, np.float64, "add", seed=1)
    q, x = torch.from_numpy(v.copy()).cuda(), torch.zeros(g.Ngather, dtype=torch.float64, device="cuda")
    g.GatherScatter(q.clone(), 1, ogs.Add, ogs.Sym)
    torch.cuda.synchronize()
    stream, graph = C.c_void_p(), C.c_void_p()
    assert rt.cudaStreamCreate(C.byref(stream)) == 0
    assert rt.cudaStreamBeginCapture(stream, 2) == 0  # relaxed
    try:
        L = _lib.lib()
        status = {"scatter": lambda: L.ogs_scatter(g.handle, q.data_ptr(), x.data_ptr(), 1, 1, 1, None),
                  "gather": lambda: L.ogs_gather(g.handle, x.data_ptr(), q.data_ptr(), 1, 1, 0, 2, None),
                  "gather_scatter": lambda: L.ogs_gather_scatter(g.handle, q.data_ptr(), 1, 1, 0, 0, None)}[call]()
    finally:
        rt.cudaStreamEndCapture(stream, C.byref(graph))
        rt.cudaGetLastError()
        rt.cudaStreamDestroy(stream)
    assert status == _lib.OGS_EDEVICE
    g.GatherScatter(q, 1, ogs.Add, ogs.Sym)
    torch.cuda.synchronize()
    ref = oracle_mod.OracleOgs(ids.copy(), "signed", unique=True)
    assert same_bits(q.cpu().numpy(), ref.gather_scatter(v.copy(), 1, "add", "sym"))
