"""The FP64 build's own reciprocal, quotient, root, logarithm and Exner powers
against 113-bit arithmetic, its bit comparisons and limiter helpers against the
language's, and the tenth of inflate against a division, over the ranges that
fim_internal.h states.  A small library with one kernel an operation is built
from that header."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from fimocn_subx_realtime_hera_apr2020_gb300 import build as B  # noqa: E402

pytestmark = pytest.mark.gpu

LD = np.longdouble
U = 2.0 ** -53  # half a unit in the last place, relative, at most
SRC = r"""
#include "fim_internal.h"
using namespace fim;
#define UNARY(NAME, T, EXPR) \
  __global__ void k_##NAME(const T* a, T* r, int n) { \
    const int q = blockIdx.x * blockDim.x + threadIdx.x; \
    if (q < n) { const T x = a[q]; r[q] = EXPR; } } \
  extern "C" int NAME(const T* a, const T*, T* r, int n) { \
    k_##NAME<<<(n + 255) / 256, 256>>>(a, r, n); return cudaDeviceSynchronize(); }
#define BINARY(NAME, T, EXPR) \
  __global__ void k_##NAME(const T* a, const T* b, T* r, int n) { \
    const int q = blockIdx.x * blockDim.x + threadIdx.x; \
    if (q < n) { const T x = a[q], y = b[q]; r[q] = EXPR; } } \
  extern "C" int NAME(const T* a, const T* b, T* r, int n) { \
    k_##NAME<<<(n + 255) / 256, 256>>>(a, b, r, n); return cudaDeviceSynchronize(); }
UNARY(t_recip, double, f64_recip(x))
UNARY(t_recip_any, double, recip(x))
BINARY(t_quot, double, f64_quot(x, y, f64_recip(y)))
BINARY(t_divide, double, divide(x, y))
UNARY(t_rsqrt, double, f64_rsqrt(x))
UNARY(t_ln, double, f64_ln13(x))
UNARY(t_pow_cp_rd, double, pow_cp_rd(x))
UNARY(t_pow_rd_cp, double, pow_rd_cp(x))
BINARY(t_lt, double, f64_lt(x, y) ? 1. : 0.)
UNARY(t_pos, double, pos(x))
UNARY(t_neg, double, neg(x))
BINARY(t_floor, double, floor_at(x, y))
BINARY(t_ratio, double, ratio01(x, y))
BINARY(t_plain_ratio, double, plain_ratio01(x, y))
BINARY(t_min0, double, min0(own_limit(x), y))
BINARY(t_min0f, float, min0(own_limit(x), y))
BINARY(t_ratiof, float, plain_ratio01(x, y))
BINARY(t_rare, double, ratio_rare(x, y) ? 1. : 0.)
BINARY(t_raref, float, ratio_rare(x, y) ? 1.f : 0.f)
UNARY(t_below0, double, below0(x) ? 1. : 0.)
UNARY(t_tenth, float, tenth(x))
UNARY(t_tenthd, double, tenth(x))
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if np.finfo(LD).eps > 1e-30:
        pytest.skip("no 113-bit long double to compare with")
    d = tmp_path_factory.mktemp("f64")
    (d / "t.cu").write_text(SRC)
    subprocess.run([B._nvcc()] + B.ARCH + ["-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I" + B.CSRC,
                                           "-I" + B.INCLUDE, str(d / "t.cu"), "-o", str(d / "t.so"), "-lcudart"],
                   check=True, env=os.environ)
    so = ctypes.CDLL(str(d / "t.so"))

    def run(name, a, b=None, dtype=np.float64):
        a = np.ascontiguousarray(a, dtype)
        ta = torch.from_numpy(a).cuda()
        tb = torch.from_numpy(np.ascontiguousarray(b, dtype)).cuda() if b is not None else ta
        r = torch.empty_like(ta)
        torch.cuda.synchronize()
        f = getattr(so, name)
        f.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int]
        assert f(ta.data_ptr(), tb.data_ptr(), r.data_ptr(), a.size) == 0
        return r.cpu().numpy()

    return run


def _log_uniform(rng, lo, hi, n):
    """Magnitudes of 2^lo .. 2^hi, all 53 bits of the fraction."""
    return rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(lo, hi, n).astype(np.float64)


def _err(got, want):
    return float(np.max(np.abs(got.astype(LD) - want) / np.abs(want)))


N = 200000


def test_reciprocal_and_quotient(lib):
    """Third-order steps from an approximation good to 2^-19: a rounding and the
    error cubed.  Quotient: one rounding, the correction's own error 2^-50 of it."""
    rng = np.random.default_rng(1)
    b = np.concatenate([_log_uniform(rng, -1000, 1000, N), 1.0 + rng.uniform(0, 1e-6, 1000), [1e-22, 1e-11, 3.0]])
    for f in ("t_recip", "t_recip_any"):
        assert _err(lib(f, b), 1 / b.astype(LD)) <= 1.125 * U, f
    a = np.concatenate([_log_uniform(rng, -400, 400, N), b[N:] * (1 + rng.uniform(-4e-16, 4e-16, 1003))])
    b = np.concatenate([_log_uniform(rng, -500, 500, N), b[N:]])
    for f in ("t_quot", "t_divide"):
        got = lib(f, a, b)
        assert _err(got, a.astype(LD) / b.astype(LD)) <= (1 + 2.0 ** -20) * U, f
        # the same as the division but for quotients half-way between two doubles
        assert np.mean(got != a / b) <= 1e-4, f


def test_divisions_without_a_number(lib):
    v = np.array([0.0, 1.0, -2.5, 1e300, np.inf, -np.inf, np.nan, -0.0])
    a, b = (x.ravel() for x in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        want, r = a / b, 1 / b
    got = lib("t_divide", a, b)
    assert np.array_equal(np.nan_to_num(got, nan=7.0), np.nan_to_num(want, nan=7.0))
    got = lib("t_recip_any", b)
    assert np.array_equal(np.nan_to_num(got, nan=7.0), np.nan_to_num(r, nan=7.0))


def test_root(lib):
    """One rounding of x r, halved by the step, the last rounding, the error cubed."""
    rng = np.random.default_rng(2)
    x = np.concatenate([_log_uniform(rng, -900, 900, N), rng.uniform(3.6e-5, 4e4, N)])
    assert _err(lib("t_rsqrt", x), 1 / np.sqrt(x.astype(LD))) <= 1.6 * U


def test_logarithm_and_powers(lib):
    """x^(cp/rd): the last rounding and 0.15 for the small power; x^(rd/cp): nine
    roundings of v^7 / x^2, a seventh of which enter, the last one, 0.2 for the
    series.  Outside 2^-20 .. 2^20 CUDA's pow (2 ulp)."""
    rng = np.random.default_rng(3)
    x = np.concatenate([_log_uniform(rng, -20, 20, 50000), rng.uniform(1e-4, 1.2, 50000),
                        [2.0 ** -20, np.nextafter(2.0 ** 20, 0), 1.0, np.nextafter(1.0, 0), np.nextafter(1.0, 2)]])
    assert np.max(np.abs(lib("t_ln", x).astype(LD) - np.log(x.astype(LD)))) <= 1e-13
    cp, rd = 1004.6855, 287.0586
    assert _err(lib("t_pow_cp_rd", x), x.astype(LD) ** LD(cp / rd)) <= 1.2 * U
    assert _err(lib("t_pow_rd_cp", x), x.astype(LD) ** LD(rd / cp)) <= 2.6 * U
    out = np.concatenate([_log_uniform(rng, -60, -20, 500), _log_uniform(rng, 20, 60, 500)])
    assert _err(lib("t_pow_cp_rd", out), out.astype(LD) ** LD(cp / rd)) <= 4 * U
    assert _err(lib("t_pow_rd_cp", out), out.astype(LD) ** LD(rd / cp)) <= 4 * U
    v = np.array([0.0, np.inf, np.nan, -1.0])
    with np.errstate(all="ignore"):
        assert np.array_equal(np.nan_to_num(lib("t_pow_rd_cp", v), nan=7.0), np.nan_to_num(v ** (rd / cp), nan=7.0))


def _specials():
    rng = np.random.default_rng(4)
    neg_nan = np.array([0xfff8 << 48], np.uint64).view(np.float64)
    v = np.concatenate([[0.0, 5e-324, -5e-324, 1e-11, 1.0, -1.0, 1e308, -1e308, np.inf, -np.inf, np.nan], neg_nan,
                        rng.normal(size=40), _log_uniform(rng, -300, 300, 20)])
    return tuple(x.ravel() for x in np.meshgrid(v, v))


def test_comparisons(lib):
    a, b = _specials()
    assert np.array_equal(lib("t_lt", a, b) != 0, a < b)
    same = lambda g, w: np.array_equal(np.nan_to_num(g, nan=7.5), np.nan_to_num(w, nan=7.5))  # noqa: E731
    assert same(lib("t_pos", a), np.where(0.0 > a, 0.0, a))
    assert same(lib("t_neg", a), np.where(0.0 < a, 0.0, a))
    pick = (b > 0) & np.isfinite(b)
    assert same(lib("t_floor", a[pick], b[pick]), np.where(a[pick] > b[pick], a[pick], b[pick]))


def test_limiter_quotients(lib):
    rng = np.random.default_rng(5)
    a = np.concatenate([rng.normal(size=N) * 2.0 ** rng.integers(-80, 80, N), [0.0, 1e300, -1e300]])
    b = np.maximum(1e-11, np.concatenate([rng.uniform(0, 2, N) * 2.0 ** rng.integers(-80, 80, N), [1.0, 1e-11, 1.0]]))
    want = np.clip(a.astype(LD) / b.astype(LD), 0, 1)
    got = lib("t_ratio", a, b)
    assert np.all(np.abs(got - want) <= want * LD((1 + 2.0 ** -20) * U))
    a, b = _specials()
    for f, dt in (("t_plain_ratio", np.float64), ("t_ratiof", np.float32)):
        with np.errstate(all="ignore"):
            x, y = a.astype(dt), b.astype(dt)
            d = np.where(y > dt(1e-11), y, dt(1e-11))
            q = x / d
            q = np.where(dt(1) < q, dt(1), q)
            q = np.where(dt(0) > q, dt(0), q)
        got = lib(f, x, y, dtype=dt)
        keep = np.ones(len(q), bool) if dt is np.float64 else ~(np.abs(d) > 2.0 ** 126)
        assert np.array_equal(np.isnan(got[keep]), np.isnan(q[keep])), f
        assert np.all(np.signbit(got[np.isnan(got)])), f  # min0 knows a NaN by its sign
        assert np.allclose(got[keep], q[keep], rtol=4e-7 if dt is np.float32 else 3e-16,
                           atol=1e-37 if dt is np.float32 else 0, equal_nan=True), f
    # a numerator that is no number, or two that cancel or add to an infinity
    with np.errstate(all="ignore"):
        for f, dt in (("t_rare", np.float64), ("t_raref", np.float32)):
            x, y = a.astype(dt), b.astype(dt)
            rare = lib(f, x, y, dtype=dt) != 0
            assert rare[~(np.isfinite(x) & np.isfinite(y))].all() and not rare[np.isfinite(x + y)].any(), f
    x = np.concatenate([a[~np.isnan(a)], [0.0, -0.0]])  # (a NaN flux's limiters do not matter)
    assert np.array_equal(lib("t_below0", x) != 0, x < 0)
    r = np.concatenate([rng.uniform(0, 1, 30), [0.0, 1.0], np.array([0xfff8 << 48], np.uint64).view(np.float64)])
    x, y = (v.ravel() for v in np.meshgrid(r, r))
    assert np.array_equal(np.nan_to_num(lib("t_min0", x, y), nan=7.5),
                          np.nan_to_num(np.where(x < y, x, y), nan=7.5))
    xf, yf = x.astype(np.float32), y.astype(np.float32)
    assert np.array_equal(np.nan_to_num(lib("t_min0f", xf, yf, dtype=np.float32), nan=7.5),
                          np.nan_to_num(np.where(xf < yf, xf, yf), nan=7.5))


def test_tenth(lib):
    """x / 10 rounded as the division, for every FP32 fraction."""
    x = (np.arange(2 ** 23, dtype=np.uint32) | 0x3f800000).view(np.float32)
    assert np.array_equal(lib("t_tenth", x, dtype=np.float32), x / np.float32(10))
    x = _log_uniform(np.random.default_rng(6), -60, 60, N)
    assert np.array_equal(lib("t_tenthd", x), x / 10)
