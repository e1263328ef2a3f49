"""The fixed-point arithmetic of the FP64 rate passes (csrc/fixp.cuh, compiled
here for the host) against wider arithmetic: products of split values, the
conversion from doubles, the exponential on its cells' edges and at random
arguments, and sums of exponentials of very different sizes."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

mpmath = pytest.importorskip("mpmath")

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "metallic_glasses_gb300", "csrc")
HARNESS = r"""
#include "fixp.cuh"
using namespace stz;
static FxExp tab[kFxExpCells];
extern "C" void t_init() { fx_exp_table(tab); }
extern "C" void t_exp(const uint64_t* Y, double* out, long n) {
  for (long i = 0; i < n; i++) out[i] = fx_double(fx_exp2_bits(Y[i], tab[fx_exp_cell(Y[i])]));
}
extern "C" void t_sum(const uint64_t* Y, double* out, long n) {
  for (long i = 0; i < n; i++) {
    FxExp c[4];
    for (int q = 0; q < 4; q++) c[q] = tab[fx_exp_cell(Y[4 * i + q])];
    out[2 * i] = fx_double(fx_exp2_sum_bits<2>(Y + 4 * i, c));
    out[2 * i + 1] = fx_double(fx_exp2_sum_bits<4>(Y + 4 * i, c));
  }
}
extern "C" void t_mad(const int64_t* x, const int64_t* y, int64_t* out, int k) {
  FxAcc a{0, 0};
  for (int i = 0; i < k; i++) fx_mad(a, fx_split(x[i]), fx_split(y[i]));
  *out = fx_value<5>(a);
}
extern "C" int t_from(double x, int s, int64_t* out) {
  bool ok = true;
  *out = fx_from_f64<4>(x, s, &ok);
  return ok;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("fixp")
    src = d / "harness.cpp"
    src.write_text(HARNESS)
    so = d / "libfixp.so"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, "-I",
                    os.path.join(cuda, "include"), str(src), os.path.join(CSRC, "fixp.cpp"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.t_from.argtypes = [C.c_double, C.c_int, C.c_void_p]
    lib.t_init()
    return lib


def _exp2(Y):
    with mpmath.workprec(160):
        return mpmath.mpf(2) ** (mpmath.mpf(int(Y)) / 2 ** 53 - 1022)


def _ulps(got, want):
    with mpmath.workprec(160):
        return abs(float((mpmath.mpf(float(got)) - want) / mpmath.ldexp(1, int(mpmath.floor(mpmath.log(want, 2))) - 52)))


def test_exponential_within_an_ulp(lib):
    rng = np.random.default_rng(1)
    cells = rng.integers(0, 2048, 400, dtype=np.uint64) << np.uint64(42)
    Y = [cells, cells + np.uint64((1 << 42) - 1), cells + np.uint64(1 << 41),
         (rng.integers(1, 2046, 1500, dtype=np.uint64) << np.uint64(53)) | rng.integers(0, 1 << 53, 1500, dtype=np.uint64)]
    Y[:3] = [(rng.integers(900, 1100, 400, dtype=np.uint64) << np.uint64(53)) + y for y in Y[:3]]
    Y = np.concatenate(Y)
    out = np.empty(len(Y))
    lib.t_exp(Y.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p), C.c_long(len(Y)))
    assert max(_ulps(o, _exp2(y)) for o, y in zip(out, Y)) < 0.9


@pytest.mark.parametrize("spread", [1, 5, 60, 300])
def test_sums_of_exponentials(lib, spread):
    """Two and four exponentials over `spread` binades: one rounding (half an
    ulp), the exponentials' own 2^-57 and the cut of 2^-60 of the largest."""
    rng = np.random.default_rng(spread)
    Y = (rng.integers(1000 - spread, 1000, (300, 4), dtype=np.uint64) << np.uint64(53)) | rng.integers(
        0, 1 << 53, (300, 4), dtype=np.uint64)
    out = np.empty((300, 2))
    lib.t_sum(Y.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p), C.c_long(300))
    for o, y in zip(out, Y):
        e = [_exp2(v) for v in y]
        with mpmath.workprec(160):
            two, four = e[0] + e[1], e[0] + e[1] + e[2] + e[3]
        assert _ulps(o[0], two) < 0.9 and _ulps(o[1], four) < 0.9


def test_products_and_conversion(lib):
    rng = np.random.default_rng(3)
    for k in (1, 5):
        for edge in (0, 1):
            x = rng.integers(-2 ** 60, 2 ** 60, k, dtype=np.int64)
            y = rng.integers(-2 ** 58, 2 ** 58, k, dtype=np.int64)
            if edge:
                x[:], y[:] = 2 ** 60 - 1, -(2 ** 58) + 1
            out = np.empty(1, np.int64)
            lib.t_mad(x.ctypes.data_as(C.c_void_p), y.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p), k)
            exact = sum(int(a) * int(b) for a, b in zip(x, y)) / 2 ** 59  # 2^5 / 2^64
            # the dropped l l products: below 2^62 / 2^64 2^5 each, and one floor
            assert abs(int(out[0]) - exact) <= 8 * k + 1
    v = np.empty(1, np.int64)
    p = v.ctypes.data_as(C.c_void_p)
    for x in (0.0, -0.0, 1.0, -1.0, 0.1, -3.7, 2.0 ** -70, -(2.0 ** -1060), 31.999):
        assert lib.t_from(x, 54, p) == 1
        want = int(mpmath.mpf(abs(x)) * 2 ** 54)
        assert int(v[0]) == (want if x >= 0 else -want)
    for x in (32.0, -32.0, 1e300, float("inf"), float("-inf"), float("nan")):
        assert lib.t_from(x, 54, p) == 0


@pytest.mark.parametrize("n", [1, 2, 3, 4, 6, 9, 16, 18, 27, 54, 72, 243, 256, 486, 648, 729, 972, 1024, 1296, 8192])
def test_twiddles_rounded_to_nearest(tmp_path, n):
    """exp(-2 pi i k / n) in 2^-62: halves put together are the nearest integers
    (a low half of -2^31 counts one up), the exact values of quarter turns
    among them."""
    src, so = tmp_path / "tw.cpp", tmp_path / "libtw.so"
    src.write_text('#include "fixp.cuh"\nextern "C" void t_tw(int n, stz::FxTwiddle* t) { stz::fx_twiddles(n, n, t); }\n')
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-I", os.path.join(cuda, "include"),
                    str(src), os.path.join(CSRC, "fixp.cpp"), "-o", str(so)], check=True)
    t = np.empty((n, 4), np.int32)
    C.CDLL(str(so)).t_tw(n, t.ctypes.data_as(C.c_void_p))
    with mpmath.workprec(160):
        for k in range(0, n, 1 + n // 512):
            a = -2 * mpmath.pi * k / n
            for v, (h, l) in ((mpmath.cos(a), t[k, :2]), (mpmath.sin(a), t[k, 2:])):
                err = abs(mpmath.mpf(int(h) * 2 ** 32 + int(l)) - v * 2 ** 62)
                assert err <= 0.5 + 1e-9 or (l == 1 - 2 ** 31 and err <= 1.5)
