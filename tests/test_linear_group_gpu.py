"""gradc::linear_group gives, whichever of its outputs a program uses, the gradients of the layers taken one by one
(the reference composes them from separate matmul nodes, frontend/tensor_math.hpp:375)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu


def test_unused_outputs_of_a_group_cost_no_gradient(tmp_path):
    exe, pkg = str(tmp_path / "linear_group_check"), os.path.join(ROOT, "gradcraft_b200")
    cmd = ["g++", "-std=c++20", "-O1", "-I", pkg, "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "linear_group_check.cpp"), "-o", exe, "-L" + pkg, "-lgradc_b200",
           "-L/usr/local/cuda/lib64", "-lcudart", "-pthread", "-Wl,-rpath," + pkg, "-Wl,-rpath,/usr/local/cuda/lib64"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    rows = [line.split() for line in r.stdout.splitlines()]
    assert [int(x[0]) for x in rows] == list(range(1, 8))
    for used, one_by_one, together, worst in rows:
        members = sum(3 << (2 + 2 * i) for i in range(3) if int(used) >> i & 1)
        assert int(one_by_one) == 3 + members  # weight and bias of the layer in front and of every layer used
        assert int(together) == int(one_by_one), used
        assert float(worst) < 1e-5, (used, worst)
