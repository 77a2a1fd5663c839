"""Allocation failures of Setup at sizes where its scratch is one block
(ogs_dsetup.cu): each is OGS_ENOMEM and leaves nothing behind."""
import ctypes as C

import pytest

from dawgs_gb300 import _lib, mesh
from test_gpu_alloc_failures import each_failure

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,unique", [(0, 0), (1, 0), (1, 1)])
@pytest.mark.parametrize("side,p", [(9, 3), (8, 10)])  # 46,656 nodes; 681,472, most of them lone
def test_block_of_scratch(cuda, side, p, kind, unique):
    L = _lib.lib()
    ids = mesh.box_ids(side, side, side, p)
    assert ids.size >= 32768
    h = C.c_void_p()

    def call():
        a = ids.copy()
        return L.ogs_setup_ex(C.byref(h), a.size, a.ctypes.data, kind, unique, _lib.SETUP_DEVICE_MAPS)
    assert each_failure(L, call, lambda: L.ogs_free(h)) >= 2  # the block and the maps' arena
