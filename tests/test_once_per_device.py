"""The kernels' shared-memory opt-in: an error is not remembered (falcon_gb300/csrc/once_per_device.h)."""
import os
import re
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "falcon_gb300", "csrc")


def test_a_failed_set_up_is_tried_again(tmp_path):
    exe = str(tmp_path / "once")
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(HERE, "once_per_device_host.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0


def test_no_launcher_keeps_an_opt_ins_error():
    for name in os.listdir(CSRC):
        text = open(os.path.join(CSRC, name)).read()
        assert not re.search(r"static\s+(const\s+)?cudaError_t", text), name
