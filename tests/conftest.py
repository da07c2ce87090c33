import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


def cuda_available() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(scope="session")
def ref():
    """The reference CPU build (oracle/_ref), or skip when it was not built."""
    from oracle import ref as R
    if not R.available():
        pytest.skip("oracle/_ref not built (needs the reference sources)")
    return R


@pytest.fixture(scope="session")
def kernel_checks(tmp_path_factory):
    """tests/cpp/kernel_checks.cu, built against the library's headers and linked to it."""
    import ctypes
    import subprocess

    from method_b200 import _lib, build
    _lib.load()
    so = str(tmp_path_factory.mktemp("checks") / "kernel_checks.so")
    src = os.path.join(ROOT, "tests", "cpp", "kernel_checks.cu")
    r = subprocess.run([build.NVCC] + build.ARCH + build.COMMON +
                       ["-fmad=false", "-shared", src, "-o", so, _lib.LIB_PATH,
                        "-Xlinker", "-rpath," + os.path.dirname(_lib.LIB_PATH)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(so)
