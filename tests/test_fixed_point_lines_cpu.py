"""The fixed-point line arithmetic of FP64 handles (wv_fx.cuh), compiled with g++."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest
import scipy.fft

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


LANES = [16, 24, 32, 48, 64, 96, 128, 192, 256]
ANY = [15, 60, 192, 198, 200, 243, 250, 256, 300, 384, 500, 512, 640, 720, 768, 1000, 1024]


def _rows(kind, n, rng):
    if kind == "equal":
        return 1.2345678901 * rng.choice([-1.0, 1.0], (2, n))
    x = rng.standard_normal((2, n))
    if kind == "smooth":
        x = np.fft.irfft(np.fft.rfft(x) / (1.0 + np.arange(n // 2 + 1)), n)
    return np.ascontiguousarray(x)


def _error(got, ref):
    return float(np.sqrt(np.sum(np.abs(got - ref) ** 2) / np.sum(np.abs(ref) ** 2)))


@pytest.mark.parametrize("lanes,n", [(1, n) for n in LANES] + [(0, n) for n in ANY])
@pytest.mark.parametrize("kind", ["smooth", "white", "equal"])
def test_long_lines_are_as_exact_as_short_ones(lib, lanes, n, kind):
    """Relative L2 error against long double at most 1.7e-16, where mixed-radix FFTs in
    doubles leave 1.4e-16 to 2.5e-16: real rows in pairs, and complex lines both ways."""
    if not np.finfo(np.longdouble).eps < 1e-18:
        pytest.skip("no long double")
    rng = np.random.default_rng(n)
    ld = np.longdouble
    worst = 0.0
    for _ in range(4):
        rows = _rows(kind, n, rng)
        out = np.empty(2 * (n // 2 + 1))
        lib.real_pair(_p(rows[0]), _p(rows[1]), n, lanes, _p(out))
        worst = max(worst, _error(out[0::2].astype(ld) + 1j * out[1::2], scipy.fft.rfft(rows[0].astype(ld))))
        z = np.ascontiguousarray(rows[0] + 1j * _rows(kind, n, rng)[0])
        if kind == "equal":
            z = np.exp(2j * np.pi * rng.random(n))
        if kind == "smooth":  # a spectrum: the inverse's input
            z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
            z = np.ascontiguousarray(z / (1.0 + np.abs(np.fft.fftfreq(n, 1.0 / n))))
        got = np.empty(2 * n)
        lib.complex_line(_p(z), n, int(kind == "smooth"), lanes, _p(got))
        ref = scipy.fft.ifft(z.astype(np.clongdouble), norm="forward") if kind == "smooth" else scipy.fft.fft(z.astype(np.clongdouble))
        worst = max(worst, _error(got[0::2].astype(ld) + 1j * got[1::2], ref))
    assert worst <= 1.7e-16, worst


@pytest.mark.parametrize("n", [127, 509])
@pytest.mark.parametrize("kind", ["smooth", "white", "equal"])
def test_prime_lines_are_no_further_off_than_sums_of_doubles(lib, n, kind):
    """A prime length is one stage of O(n) sums: against the same sums in doubles."""
    if not np.finfo(np.longdouble).eps < 1e-18:
        pytest.skip("no long double")
    rng = np.random.default_rng(n)
    m = np.arange(n)
    tw = np.exp(-2j * np.pi * m / n)
    rows = _rows(kind, n, rng)
    ref = scipy.fft.rfft(rows[0].astype(np.longdouble))
    out = np.empty(2 * (n // 2 + 1))
    lib.real_pair(_p(rows[0]), _p(rows[1]), n, 0, _p(out))
    plain = np.zeros(n // 2 + 1, complex)
    for i in range(n):
        plain += rows[0][i] * tw[i * m[:n // 2 + 1] % n]
    assert _error(out[0::2].astype(np.longdouble) + 1j * out[1::2], ref) <= _error(plain, ref)


@pytest.mark.parametrize("lanes,n", [(1, n) for n in LANES] + [(0, n) for n in (60, 200, 250, 384, 500, 512, 1000, 1024)])
def test_line_sums_have_no_mean_error(lib, lanes, n):
    """The first coefficient is the sum of the entries, where a mean of the roundings would
    collect: over 400 white rows its mean error stays within five standard errors."""
    if not np.finfo(np.longdouble).eps < 1e-18:
        pytest.skip("no long double")
    rng = np.random.default_rng(7 * n)
    error = []
    for _ in range(400):
        rows = rng.standard_normal((2, n))
        out = np.empty(2 * (n // 2 + 1))
        lib.real_pair(_p(rows[0]), _p(rows[1]), n, lanes, _p(out))
        error.append(float(out[0] - np.sum(rows[0].astype(np.longdouble))))
    assert abs(np.mean(error)) <= 5.0 * np.std(error) / 20.0, (np.mean(error), np.std(error))


@pytest.mark.parametrize("lanes,n", [(1, 128), (1, 192), (1, 256)] + [(0, n) for n in (200, 251, 256, 384, 500, 509, 512, 1000, 1024)])
def test_equal_moduli_at_the_exponent_boundary(lib, lanes, n):
    """Equal moduli near a power of two of the bounds, where the float sum may round past
    n times the largest: every bit a line starts finer by has to come down again."""
    rng = np.random.default_rng(n)
    sign = rng.choice([-1.0, 1.0], (2, n))
    ref = np.fft.rfft(sign[0])
    out = np.empty(2 * (n // 2 + 1))
    boundary = 2.0 ** np.arange(3) / 1.0025
    for c in np.concatenate([b * (1.0 + np.arange(-120, 121) * 2.0 ** -23) for b in boundary]):
        rows = np.ascontiguousarray(c * sign)
        lib.real_pair(_p(rows[0]), _p(rows[1]), n, lanes, _p(out))
        assert _error(out[0::2] + 1j * out[1::2], c * ref) <= 1e-15, c
