"""Function attributes and device properties are kept per device: what one device was told or
asked says nothing about the next."""
import glob
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "caffe_old_b200", "csrc")


def test_one_answer_per_device(tmp_path):
    exe = str(tmp_path / "per_device")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, os.path.join(HERE, "cpp", "per_device.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.stdout == "1 1 1 wrong 0 beyond 2\n"


def test_every_function_attribute_is_set_per_device():
    """Each cudaFuncSetAttribute stands inside a PerDevice answer: no static of its own says that it was done."""
    calls = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        src = open(path).read()
        for m in re.finditer(r"cudaFuncSetAttribute\(", src):
            calls += 1
            before = src[:m.start()]
            assert ".get(current_device(), " in before[before.rindex("PerDevice<"):], (os.path.basename(path), before.count("\n") + 1)
    assert calls > 0
