"""The f64 min-sum scaling by integer products (csrc/scale_f64.cuh) on the host, where its
copy runs the same operations: bit for bit the processor's multiplication."""

import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_integer_products_round_as_the_multiplication(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ is needed")
    exe = str(tmp_path / "scale_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "native", "scale_check.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
