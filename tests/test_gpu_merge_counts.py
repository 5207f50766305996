"""The merge reads only candidate lists whose length the fused pass can have
written (tests/cpp/test_merge_counts.cpp): the rule on the host, the merge over
lengths that break it on a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(tmp_path, *args):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe, lib = str(tmp_path / "tm"), os.path.join(ROOT, "curplsh_b200")
    r = subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-x", "cu",
                        "-I", os.path.join(lib, "csrc"), os.path.join(ROOT, "tests", "cpp", "test_merge_counts.cpp"),
                        "-L", lib, "-lcurplsh_b200", "-Xlinker", f"-rpath={lib}", "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, *args], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "merge counts ok" in r.stdout, r.stdout + r.stderr


def test_list_lengths_the_merge_reads(tmp_path):
    _run(tmp_path)


@pytest.mark.gpu
def test_merge_skips_lists_of_impossible_length(tmp_path):
    _run(tmp_path, "gpu")
