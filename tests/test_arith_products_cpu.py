"""Host check of the recursions' modular products and the bounds their lazy passes rely on."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CUDA_INC = "/usr/local/cuda/include"


def test_products_against_exact_arithmetic(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.isdir(CUDA_INC):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "arith_products")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "inspire-rs_gb300", "csrc"), "-I", CUDA_INC,
                    os.path.join(ROOT, "tests", "arith_products.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "1000000"], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
