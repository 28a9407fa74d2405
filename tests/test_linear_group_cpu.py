"""What gradc::linear_group refuses, as separate layers do (frontend/tensor_math.hpp:375)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_input_and_parameters_on_two_devices_are_refused(tmp_path):
    from gradcraft_b200 import build

    build.build()
    exe, pkg = str(tmp_path / "group_device_check"), os.path.join(ROOT, "gradcraft_b200")
    cmd = ["g++", "-std=c++20", "-O1", "-I", pkg, "-I/usr/local/cuda/include", os.path.join(ROOT, "tests", "group_device_check.cpp"), "-o", exe, "-L" + pkg, "-lgradc_b200",
           "-L/usr/local/cuda/lib64", "-lcudart", "-pthread", "-Wl,-rpath," + pkg, "-Wl,-rpath,/usr/local/cuda/lib64"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr[-2000:]
    assert r.stdout.split() == ["taken", "refused"]
