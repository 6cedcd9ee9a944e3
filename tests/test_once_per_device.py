"""A kernel's dynamic shared-memory limit belongs to the device that is current when it
is set: every launcher sets it once on each device (plum_gb300/csrc/per_device.h), here
against a fake of the call."""
import glob
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "plum_gb300", "csrc")


def test_flag_is_keyed_by_device(tmp_path):
    exe = str(tmp_path / "once")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-o", exe,
                        os.path.join(HERE, "once_per_device_harness.cc")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


def test_every_launcher_uses_it():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) +
                       glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            text = f.read()
        assert "cudaFuncSetAttribute" not in text, path
        # a call's device is selected, and known, through one function
        assert "cudaSetDevice" not in text and "cudaGetDevice(" not in text, path
        # no other state of a device in a function's or a file's static flag
        assert not re.search(r"static (bool|int) \w+ = (false|0);", text), path
        assert len(re.findall(r"\bOncePerDevice (\w+)", text)) <= len(
            re.findall(r"\ballow_smem\(", text)), path
