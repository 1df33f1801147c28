"""The choice between the one-CTA Respond kernel's two forms
(csrc/batch_policy.h) on the host: a C++
driver built with g++."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "inspire-rs_gb300", "csrc")


def test_batch_policy_on_host(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "batch_policy_check")
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", CSRC,
                    os.path.join(HERE, "native", "batch_policy_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
