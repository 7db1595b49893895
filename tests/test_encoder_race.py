"""The tensor-map encoder is found once, whichever threads ask first: a thread
that asked during the first look-up took large boxes for ones that the
tensor-copy unit cannot address (compiled against the library's host side,
without a device)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
def test_both_threads_get_the_encoder(tmp_path):
    lib = os.path.join(ROOT, "carpet_b200")
    if not os.path.exists(os.path.join(lib, "libcgx.so")):
        pytest.skip("libcgx.so is not built")
    exe = str(tmp_path / "check")
    r = subprocess.run([NVCC, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I" + os.path.join(lib, "csrc"),
                        os.path.join(ROOT, "tests", "encoder_race_check.cu"), "-L" + lib, "-lcgx",
                        "-Xlinker", "-rpath=" + lib, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
