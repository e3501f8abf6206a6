"""The ordered walk over records that are no tree ends with an error word
instead of passing what it had listed for the whole."""
import os
import shutil
import subprocess

import pytest

from conftest import HAS_GPU, PKG, ROOT

pytestmark = pytest.mark.gpu


def test_inconsistent_records(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not HAS_GPU or not os.path.exists(nvcc):
        pytest.skip("needs a CUDA device and nvcc")
    exe = str(tmp_path / "walk_records_test")
    subprocess.check_call([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "--expt-relaxed-constexpr",
                           f"-I{os.path.join(ROOT, 'include')}", f"-I{os.path.join(PKG, 'csrc')}",
                           os.path.join(ROOT, "tests", "cpp", "walk_records_test.cu"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stderr
    one, cycle, outside = [tuple(map(int, line.split())) for line in out.stdout.split("\n")[:3]]
    assert one == (1, 0)
    assert cycle == (0, 804)  # traversal stage, inconsistent topology
    assert outside == (0, 804)
