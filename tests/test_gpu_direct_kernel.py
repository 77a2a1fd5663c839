"""The direct CTA kernel for every row (-DOGS_KERNEL=2: the kernel of calls with
more components than the pipelines' arithmetic holds) against the recorded
outputs of gslib and the oracle's: those tests, run with a library built so."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_direct_kernel(cuda, oracle_mod, tmp_path):
    from dawgs_gb300 import build
    lib = str(tmp_path / "libdawgs_ogs_direct.so")
    build.build(extra=["-DOGS_KERNEL=2"], build_dir=str(tmp_path / "obj"), lib=lib)
    env = dict(os.environ, DAWGS_OGS_LIB=lib)
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider",
                        os.path.join(HERE, "test_gpu_gslib.py"), os.path.join(HERE, "test_gpu_random_parity.py")],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-3000:]
