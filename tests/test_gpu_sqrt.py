"""The kernels' FP32 square roots (csrc/phase_math.cuh) against sqrtf: every bit
pattern, so zeros, subnormals, both ends of the fast range, infinities and NaN too."""
import ctypes
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    from pystamps_b200 import build

    so = tmp_path_factory.mktemp("sqrt") / "sqrt_check.so"
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-o", str(so), str(Path(__file__).with_name("sqrt_check.cu"))],
                   check=True)
    fn = ctypes.CDLL(str(so)).sqrt_check
    fn.argtypes = [ctypes.c_uint32, ctypes.c_uint64, ctypes.c_void_p]

    def run(first, count):
        bad = (ctypes.c_uint64 * 2)()
        assert fn(first, count, bad) == 0
        return list(bad)

    return run


@pytest.mark.parametrize("first", [k << 28 for k in range(16)])
def test_every_float(check, first):
    assert check(first, 1 << 28) == [0, 0]


# 0, the largest subnormal, 2^-100, infinity, the largest NaN, -0
@pytest.mark.parametrize("pattern", [0, 0x007FFFFF, 0x0D800000, 0x7F800000, 0x7FFFFFFE, 0x80000000])
def test_edges(check, pattern):
    assert check(max(pattern - 2, 0), 4) == [0, 0]
