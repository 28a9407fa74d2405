"""Generation refuses a model that does not lie on the inference device, as the reference's forward does
(GPTGenerator::run_inference, nn/generators/gpt_generator.hpp:12-132), and takes it once it has been moved."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


def test_a_model_elsewhere_is_refused(tmp_path):
    exe, pkg = str(tmp_path / "generation_device_check"), os.path.join(ROOT, "gradcraft_b200")
    cmd = ["g++", "-std=c++20", "-O1", "-I", pkg, "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "generation_device_check.cpp"), "-o", exe, "-L" + pkg, "-lgradc_b200",
           "-L/usr/local/cuda/lib64", "-lcudart", "-pthread", "-Wl,-rpath," + pkg, "-Wl,-rpath,/usr/local/cuda/lib64"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    refused, taken = r.stdout.splitlines()
    assert "same device" in refused and taken == "12"
