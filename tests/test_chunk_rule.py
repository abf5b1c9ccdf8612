"""The work chunk of a call (``effective_chunk`` in ``csrc/pds_internal.h``), compiled for the host:
the autotuner's first candidate is the library default, so the chunk it names must get the
default's rule (up to 8192 photons while 48 chunks an SM are left), and chunks that are not the
default keep their size."""
import os
import shutil
import subprocess

import pytest

from shapefromcaustics_b200 import autotune

HERE = os.path.dirname(os.path.abspath(__file__))
SMS = 148


def _nvcc():
    p = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    return p if os.path.exists(p) else shutil.which("nvcc")


@pytest.mark.skipif(_nvcc() is None, reason="nvcc not found")
def test_chunks(tmp_path):
    exe = str(tmp_path / "chunk_rule_check")
    subprocess.check_call([_nvcc(), "-std=c++17", os.path.join(HERE, "chunk_rule_check.cu"), "-o", exe])
    default = autotune.DEFAULT["chunk"]
    cases = [(default, 1, 256), (default, 2 ** 20, 768), (default, 2 ** 22, 2048),
             (default, 2048 * 48 * SMS, 2048), (default, 2048 * 48 * SMS + 1, 2304),
             (default, 2 ** 26, 8192), (default, 2 ** 30, 8192), (1024, 2 ** 26, 1024),
             (4096, 2 ** 26, 4096), (4096, 2 ** 20, 768), (2 ** 20, 2 ** 26, 37888)]
    args = [str(v) for chunk, n, _ in cases for v in (chunk, n, SMS)]
    out = subprocess.check_output([exe, *args], text=True).split()
    assert [int(v) for v in out] == [want for _, _, want in cases]
