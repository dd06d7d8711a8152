"""The bounded wait of the respond clusters: complete phases are seen, a phase that nothing completes is given up within
seconds and leaves the context usable."""
import os
import subprocess

import pytest

from conftest import ROOT, load_package

pytestmark = pytest.mark.gpu


def test_wait_gives_up(tmp_path):
    build = load_package()._build
    exe = str(tmp_path / "inbox_wait")
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I", build.CSRC, os.path.join(ROOT, "tests", "inbox_wait.cu"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip().endswith("ok"), out.stdout + out.stderr
