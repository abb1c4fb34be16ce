"""The arithmetic rules that the kernels share with the host (hsr_internal.h), checked on the CPU."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rules_on_the_host(tmp_path):
    import build_lib

    if not shutil.which("g++"):
        pytest.skip("no host compiler")
    cuda = os.path.dirname(os.path.dirname(build_lib.nvcc()))
    exe = tmp_path / "host_rules_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(cuda, "include"), "-I",
                    os.path.join(ROOT, "hana-softwarerenderer_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "host_rules_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


def test_a_plan_counts_what_its_clearing_views_clear():
    """A batch of several draws into one target clears it once (the first draw); the others' empty tiles
    are not to be cleared."""
    src = open(os.path.join(ROOT, "hana-softwarerenderer_gb300", "csrc", "hsr_runtime.cu")).read()
    assert re.search(r"if \(d\.flags & HSR_DRAW_CLEAR\) \{\s*p\.clear_bytes \+=", src)
    assert src.count("clear_bytes +=") == 1
