"""Kernel attributes are set once per device, not once per process (DeviceOnce of
device_once.h, which every launch of a kernel with attributes goes through).  No GPU."""
import glob
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "utr_public_gb300", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_once_per_device(tmp_path):
    exe = str(tmp_path / "device_once_host")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I" + CSRC,
                    os.path.join(ROOT, "tests", "device_once_host.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["1", "1", "1", "3", "0"]


def test_attributes_are_set_through_it():
    """No launch code keeps its attributes behind a flag of the process."""
    for path in glob.glob(os.path.join(CSRC, "*launch.cuh")):
        text = open(path).read()
        assert "once_flag" not in text, path
        for m in re.finditer(r"cudaFuncSetAttribute\(", text):
            assert re.search(r"(once|f)\.run\(current_device\(\)", text[max(0, m.start() - 700):m.start()]), path
