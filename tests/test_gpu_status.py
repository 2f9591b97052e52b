"""GPU: the device status of a count reaches the caller (tests/compat/status_check.cu, which sets it by hand)."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def build(out):
    from miniisosurface_gb300 import builder

    d = builder.library_path().parent
    res = subprocess.run([builder.nvcc_path(), *builder.ARCH, "-std=c++17", "-I", str(ROOT / "include"),
                          str(ROOT / "tests" / "compat" / "status_check.cu"), "-o", str(out), "-L", str(d), "-lminiiso",
                          "-Xlinker", "-rpath", "-Xlinker", str(d)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout + res.stderr
    return out


def test_status_check_compiles(built, tmp_path):
    assert build(tmp_path / "status_check").exists()


@pytest.mark.gpu
def test_status_reaches_the_caller(cuda, tmp_path):
    res = subprocess.run([str(build(tmp_path / "status_check"))], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
