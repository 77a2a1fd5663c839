"""The checked build (-DOGS_CHECK_BOUNDS=1) on handles with lone tiles whose node
count ends within a word and within a tile: it finds no id out of range, and the
results are the oracle's, bit for bit."""
import json
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = textwrap.dedent('''
    import json
    import numpy as np, torch
    import oracle
    from dawgs_gb300 import ogs
    from helpers import same_bits, values
    from test_gpu_lone_tiles import mostly_lone

    out = {}
    for n in (515, 4100, 70003, 4000003):
        base = mostly_lone(n, seed=n)
        for kind, un in (("unsigned", False), ("signed", True)):
            g = ogs.ogs_t().Setup(n, base.copy(), None, ogs.Signed if un else ogs.Unsigned, ogs.Auto, un)
            ref = oracle.OracleOgs(base.copy(), kind, unique=un)
            ok = True
            for dt in (np.float64, np.float32):
                v = values(n, dt, "add", seed=3)
                for op, oname in ((ogs.Add, "add"), (ogs.Max, "max")):
                    d = torch.from_numpy(v.copy()).cuda()
                    g.GatherScatter(d, 1, op, ogs.Sym)
                    ok &= same_bits(d.cpu().numpy(), ref.gather_scatter(v.copy(), 1, oname, "sym"))
                if un:
                    gv = torch.zeros(g.Ngather, dtype=d.dtype, device="cuda")
                    g.Gather(gv, torch.from_numpy(v.copy()).cuda(), 1, ogs.Add, ogs.Trans)
                    ok &= same_bits(gv.cpu().numpy(), ref.gather(np.zeros(g.Ngather, dt), v.copy(), 1, "add", "trans"))
            torch.cuda.synchronize()
            out[f"{kind} {n}"] = [g.checked_id_errors(), bool(ok)]
    print(json.dumps(out))
''')


def test_checked_build_on_lone_tiles(cuda, oracle_mod, tmp_path):
    from dawgs_gb300 import build
    lib = str(tmp_path / "libdawgs_ogs_checked.so")
    build.build(extra=["-DOGS_CHECK_BOUNDS=1"], build_dir=str(tmp_path / "obj"), lib=lib)
    env = dict(os.environ, DAWGS_OGS_LIB=lib,
               PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests"), os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=ROOT, env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    res = json.loads(r.stdout.strip().splitlines()[-1])
    assert len(res) == 8
    assert all(v == [0, True] for v in res.values()), res
