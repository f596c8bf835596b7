"""The fixed-point line arithmetic of FP64 handles (wv_fx.cuh), compiled with g++."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    so = str(tmp_path_factory.mktemp("fx") / "fixed_point_lines.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC",
                           f"-I{ROOT}/wave-vortex-model_gb300/csrc", f"-I{ROOT}/include",
                           os.path.join(ROOT, "tests", "fixed_point_lines.cpp"),
                           os.path.join(ROOT, "wave-vortex-model_gb300", "csrc", "wv_plan.cpp"),
                           os.path.join(ROOT, "wave-vortex-model_gb300", "csrc", "wv_descriptor.cpp"), "-o", so])
    return ctypes.CDLL(so)


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.mark.parametrize("sh", [0, 1, 2, 3, 9, 40, 63])
def test_aligned_products_round_without_a_mean(lib, sh):
    """Within half a unit each, and a mean below 5 standard errors of 2^20 values that
    are uniform in the unit (0.29 / 2^10 units), ties at a shift of one included."""
    rng = np.random.default_rng(3)
    n = 1 << 20
    x = rng.integers(-(1 << 61), 1 << 61, n, dtype=np.int64)
    out = np.empty_like(x)
    lib.align_products(_p(x), ctypes.c_size_t(n), ctypes.c_int(sh), _p(out))
    if sh == 63:
        assert not out.any()
        return
    error = (out.astype(object) * (1 << sh) - x.astype(object)).astype(np.float64) / (1 << sh)
    assert np.max(np.abs(error)) <= 0.5
    assert abs(np.mean(error)) <= 5 * 0.29 / 2 ** 10 + (0.25 * 5 / 2 ** 10 if sh == 1 else 0.0)


@pytest.mark.parametrize("sh", [-9, 0, 1, 2, 3, 5, 9])
def test_shifted_products_round_without_a_mean(lib, sh):
    """As above: one tie in 2^sh rounded up every time was 2^-(sh + 1) units of mean, which
    put 5.7e-13 instead of 2e-14 on F0 of the horizontal mean at 16x384x9."""
    rng = np.random.default_rng(4)
    n = 1 << 20
    x = rng.integers(-(1 << 48), 1 << 48, n, dtype=np.int64)
    out = np.empty_like(x)
    lib.shift_products(_p(x), ctypes.c_size_t(n), ctypes.c_int(sh), _p(out))
    if sh <= 0:
        assert np.array_equal(out, x << -sh)
        return
    error = (out * (1 << sh) - x) / (1 << sh)
    assert np.max(np.abs(error)) <= 0.5
    assert abs(np.mean(error)) <= 5 * 0.36 / 2 ** 10
