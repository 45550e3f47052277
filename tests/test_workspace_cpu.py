"""The MATVEC workspace after a failed allocation, on CPU: half a workspace must not
pass for a complete one (the next MATVEC would run on a null slab)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "ddscat-cuda_b200")
OBJ = [os.path.join(PKG, "build", n) for n in ("matvec.o", "matvec_x.o")]

pytestmark = pytest.mark.skipif(shutil.which("nvcc") is None or not all(os.path.exists(o) for o in OBJ),
                                reason="nvcc or the library's objects not available")


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("workspace") / "driver")
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-o", exe, os.path.join(ROOT, "tests", "workspace_driver.cu"),
                    *OBJ], check=True, capture_output=True, text=True)
    return exe


def _calls(driver, fail):
    out = subprocess.run([driver, str(fail)], check=True, capture_output=True, text=True).stdout
    return [tuple(int(v) for v in line.split()) for line in out.splitlines()]


@pytest.mark.parametrize("fail", [1, 2])
def test_failed_workspace_is_dropped_and_built_again(driver, fail):
    size = (2 * 3 * 8 * 16 * 8 + 2 * 16 * 3 * 16 * 8) * 8  # A and B of two right-hand sides
    first, second = _calls(driver, fail)
    assert first == (1, 0, 0, 0, 0)
    assert second == (0, 1, 1, 2, size)


def test_workspace_is_kept(driver):
    first, second = _calls(driver, 0)
    assert first == second and first[:4] == (0, 1, 1, 2)
