"""reciprocal() of the strip kernels against the division, on the device.  The
result is within 1/2 + 2^-7 ulp of 1/d: the correctly rounded value or, where
1/d lies within 2^-7 ulp of the middle between two numbers (a part of 2^-6 of
all d at most; bar twice that), its neighbour."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = "/usr/local/cuda/bin/nvcc"


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n", [("0", 1 << 26), ("1", 1 << 26), ("2", 64 * 2041)])
def test_reciprocal(tmp_path, kind, n):
    if not os.path.exists(NVCC):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "reciprocal")
    subprocess.check_call([NVCC, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a",
                           "--expt-relaxed-constexpr", "-o", exe,
                           os.path.join(HERE, "device", "reciprocal.cu")])
    state, differ, most = subprocess.check_output([exe, kind, str(n)]).decode().rsplit(None, 2)
    assert state == "no error"
    assert int(most) <= 1, most
    if kind != "2":
        assert int(differ) <= n / 32, differ
