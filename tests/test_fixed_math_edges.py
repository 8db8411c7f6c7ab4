"""The integer-arithmetic sin, cos, exp, log and tanh (csrc/fixed_math.cuh, compiled for the host) at the
ends of their ranges and where one of their formulas takes over from another.

Bounds in ulps: 0.5 for the rounding to double, and the fixed-point result's own error: interpolants
within 2^-57 of the result, 1/16 ulp; tanh from 1/8 on is a quotient of 64-bit numbers at the end of a
chain of truncated products, off by up to 8 units of 2^-62 where the result is as small as 1/8 (ulp
2^-56), 1/8 ulp."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "casadi_gb300",
                    "csrc")
SHIM = r"""
#include "fixed_math.cuh"
using namespace cgb;
template <class F> static void each(int n, const double* x, double* r, unsigned char* took, F f) {
  for (int i = 0; i < n; ++i) { r[i] = 7.25; took[i] = f(x[i], r + i) ? 1 : 0; }
}
extern "C" {
void t_exp(int n, const double* x, double* r, unsigned char* k) { each(n, x, r, k, fx_exp); }
void t_log(int n, const double* x, double* r, unsigned char* k) { each(n, x, r, k, fx_log); }
void t_tanh(int n, const double* x, double* r, unsigned char* k) { each(n, x, r, k, fx_tanh); }
void t_sqrt(int n, const double* x, double* r, unsigned char* k) { each(n, x, r, k, fx_sqrt); }
void t_sin(int n, const double* x, double* r, unsigned char* k) {
  each(n, x, r, k, [](double v, double* s) { double c; return fx_sincos(v, s, &c); });
}
void t_cos(int n, const double* x, double* r, unsigned char* k) {
  each(n, x, r, k, [](double v, double* c) { double s; return fx_sincos(v, &s, c); });
}
}
"""
BOUND = {"sin": "0.5625", "cos": "0.5625", "exp": "0.5625", "log": "0.5625", "tanh": "0.625"}


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("fxe")
    (d / "fx.cpp").write_text(SHIM)
    so = str(d / "fx.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    CSRC, str(d / "fx.cpp"), "-o", so], check=True)
    lib = ct.CDLL(so)

    def call(name, x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        out, took = np.empty(x.size), np.empty(x.size, np.uint8)
        getattr(lib, "t_" + name)(x.size, *[ct.c_void_p(a.ctypes.data) for a in (x, out, took)])
        return out, took.astype(bool)

    return call


def around(points, rng, n=40):
    """The points, their neighbours and arguments within a few per mille of them."""
    p = np.asarray(points, dtype=np.float64)
    with np.errstate(over="ignore"):
        out = [p, np.nextafter(p, np.inf), np.nextafter(p, -np.inf)]
        out += [p * (1 + s * rng.uniform(0, 1, p.size)) for s in (1e-3, -1e-3, 1e-9, -1e-9)
                for _ in range(n // 8)]
    x = np.concatenate(out)
    return x[np.isfinite(x)]


def points(name, rng):
    if name == "exp":  # 539.3 thousandths at the last
        x = [2.0 ** -34, 2.0 ** -54, 699.9, 1.0, 0.6931471805599453, 56.144705494437972,
             260.62333989054497]
        return around(np.concatenate([x, np.negative(x), [0.0]]), rng)
    if name == "log":
        return around([1.0, 2.0 ** 0.5, 0.5 ** 0.5, 2.0, 0.5, 2.0 ** -1022, 1.7976931348623157e308,
                       1.278837678531576], rng)
    if name == "tanh":  # 611 thousandths at the last
        x = [0.125, 2.0 ** -27, 32.0, 19.0615, 22.0, 1.0, 0.12524055555695113, 0.12537959991750341]
        return around(np.concatenate([x, np.negative(x)]), rng)
    k = rng.integers(1, 20860, 60) * (np.pi / 2)  # |x| < 2^15
    return around(np.concatenate([k, -k, [0.0, 2.0 ** -33, 1.0, 32767.9, 0.95628254412940272]]), rng, 16)


@pytest.mark.parametrize("name", sorted(BOUND))
def test_every_accepted_argument_is_within_its_bound(host, name):
    mp = pytest.importorskip("mpmath")
    mp.mp.prec = 200
    x = points(name, np.random.default_rng(11))
    got, took = host(name, x)
    assert not np.isnan(got).any()
    inside = {"exp": np.abs(x) < 699, "log": x >= 2.0 ** -1022, "tanh": x == x,
              "sin": np.abs(x) < 32768, "cos": np.abs(x) < 32768}[name]
    # within 2^-24 or so of a multiple of pi/2 the reduced argument may have too few bits
    near = np.abs(np.sin(2 * x)) < 2.0 ** -22 if name in ("sin", "cos") else np.zeros(x.size, bool)
    assert (took | ~inside | near).all(), x[~took & inside & ~near][:5]
    f, worst = getattr(mp, name), mp.mpf(0)
    for g, v in zip(got[took].tolist(), x[took].tolist()):
        t = f(mp.mpf(v))
        if t == 0:
            assert g == 0
            continue
        ulp = mp.mpf(2) ** (max(mp.floor(mp.log(abs(t), 2)), -1022) - 52)
        worst = max(worst, abs(mp.mpf(g) - t) / ulp)
    assert worst <= mp.mpf(BOUND[name]), worst


@pytest.mark.parametrize("name", sorted(BOUND) + ["sqrt"])
def test_what_is_not_a_range_s_argument_is_refused(host, name):
    """Infinities and NaN are refused by every routine, and so are negative arguments of log and sqrt:
    their results are the caller's."""
    x = np.array([np.inf, -np.inf, np.nan, -np.nan])
    if name in ("log", "sqrt"):
        x = np.concatenate([x, [-1.0, -5e-324, -1e308]])
    if name == "log":
        x = np.concatenate([x, [0.0, -0.0, 5e-324]])
    _, took = host(name, x)
    assert not took.any(), x[took]
