"""The library's kernel launch over a fake of the runtime's launch call: a refused launch is returned
to the caller once and leaves no error for whoever asks the runtime next."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
INVALID_VALUE, INVALID_HANDLE, NO_KERNEL_IMAGE = 1, 400, 209


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    from p2r_tests_b200.build import cuda_home
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    so = tmp_path_factory.mktemp("launch") / "liblaunch_host.so"
    # -Bsymbolic: the fakes answer, whatever CUDA runtime the process has loaded
    subprocess.run([cxx, "-std=c++17", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I" + str(cuda_home() / "include"),
                    "-I" + str(ROOT / "p2r_tests_b200" / "csrc"), "-o", str(so),
                    str(ROOT / "tests" / "launch_host.cpp")], check=True)
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("result", [INVALID_VALUE, INVALID_HANDLE, NO_KERNEL_IMAGE])
def test_refused_launch_leaves_no_pending_error(fake, result):
    left = ctypes.c_int(-1)
    assert fake.fake_launch(result, 0, ctypes.byref(left)) == result
    assert left.value == 0


def test_accepted_launch(fake):
    left = ctypes.c_int(-1)
    assert fake.fake_launch(0, 0, ctypes.byref(left)) == 0
    assert left.value == 0
