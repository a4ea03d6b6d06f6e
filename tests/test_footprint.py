"""What the engine and the job server take a batch's device memory to be (pdpd_footprint.hpp):
bucket sizes of batches of mixed density, admission by the budget and by the reach of the FP64
pair lists, the snapshot buffers' reservation."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_footprint(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "footprint_check")
    subprocess.run([gxx, "-O1", "-std=c++17", "-Wall", "-Werror", os.path.join(HERE, "footprint_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
