"""A context's settings may change between a forward and its backward: the fused attention forward keeps row statistics (not the
probabilities that the reference's CausalSoftmax node keeps, frontend/tensor_other.hpp:53-93), so the backward then forms them."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


def test_backward_after_the_setting_has_changed(tmp_path):
    exe, pkg = str(tmp_path / "attention_setting_check"), os.path.join(ROOT, "gradcraft_b200")
    cmd = ["g++", "-std=c++20", "-O1", "-I", pkg, "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "attention_setting_check.cpp"), "-o", exe, "-L" + pkg, "-lgradc_b200",
           "-L/usr/local/cuda/lib64", "-lcudart", "-pthread", "-Wl,-rpath," + pkg, "-Wl,-rpath,/usr/local/cuda/lib64"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]
    rows = [line.split() for line in r.stdout.splitlines()]
    assert [x[0] for x in rows] == ["64", "300"]
    # the operator tests hold either path to 2e-5 (2-norm) of the float64 gradients, so the two are within twice that
    assert all(float(x[1]) < 4e-5 for x in rows), rows
