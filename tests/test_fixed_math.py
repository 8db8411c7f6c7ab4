"""The integer-arithmetic division, square root, sin/cos, exp, log and tanh of the sweeps
(csrc/fixed_math.cuh), compiled for the host and run on the GPU.

Division and square root are correctly rounded: equal to the host's bit for bit. The others are
within 0.6 ulp of the exact value: 0.5 for the final rounding to double and less than 0.1 for
truncated products and the interpolants (errors below 2^-57 of the result, ulps of 2^-53)."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

from casadi_gb300 import calculus as C
from casadi_gb300 import sx as S

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "casadi_gb300",
                    "csrc")
SHIM = r"""
#include "fixed_math.cuh"
#include <string.h>
using namespace cgb;
template <class F> static int each(int n, const double* x, double* r, F f) {
  int left = 0;
  for (int i = 0; i < n; ++i) if (!f(x[i], r + i)) { ++left; r[i] = 0.0 / 0.0; }
  return left;
}
extern "C" {
int t_div(int n, const double* x, const double* y, double* q) {
  int left = 0;
  for (int i = 0; i < n; ++i)
    if (!fx_div(x[i], fx_divisor(y[i]), q + i)) { ++left; q[i] = x[i] / y[i]; }
  return left;
}
int t_sqrt(int n, const double* x, double* r) { return each(n, x, r, fx_sqrt); }
int t_exp(int n, const double* x, double* r) { return each(n, x, r, fx_exp); }
int t_log(int n, const double* x, double* r) { return each(n, x, r, fx_log); }
int t_tanh(int n, const double* x, double* r) { return each(n, x, r, fx_tanh); }
int t_sin(int n, const double* x, double* r) {
  return each(n, x, r, [](double v, double* s) { double c; return fx_sincos(v, s, &c); });
}
int t_cos(int n, const double* x, double* r) {
  return each(n, x, r, [](double v, double* c) { double s; return fx_sincos(v, &s, c); });
}
}
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("fx")
    (d / "fx.cpp").write_text(SHIM)
    so = str(d / "fx.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    CSRC, str(d / "fx.cpp"), "-o", so], check=True)
    lib = ct.CDLL(so)

    def call(name, *xs):
        xs = [np.ascontiguousarray(x, dtype=np.float64) for x in xs]
        out = np.empty(xs[0].size)
        left = getattr(lib, "t_" + name)(xs[0].size, *[ct.c_void_p(x.ctypes.data) for x in xs],
                                         ct.c_void_p(out.ctypes.data))
        return out, left

    return call


def doubles(rng, n, lo, hi, signed=True):
    """Doubles of exponents [lo, hi) with random, short, all-ones and all-zeros mantissas."""
    m = rng.integers(0, 1 << 52, n).astype(np.uint64)
    k = rng.integers(0, 6, n)
    m[k == 0] &= np.uint64(0xFFFFFF)
    m[k == 1] &= np.uint64(0xFFFFFFF000000)
    m[k == 2] = np.uint64((1 << 52) - 1) - (m[k == 2] & np.uint64(7))
    m[k == 3] &= np.uint64(7)
    b = m | (rng.integers(lo + 1023, hi + 1023, n).astype(np.uint64) << np.uint64(52))
    if signed:
        b |= rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63)
    return b.view(np.float64).copy()


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -2.5e-310, 2.0**-1022, 1.0, -1.0,
                    1.7976931348623157e308, -3.0, 0.1])


def test_division_and_root_are_correctly_rounded(host):
    rng = np.random.default_rng(0)
    n = 400000
    with np.errstate(all="ignore"):
        for lo, hi in ((-300, 300), (-1022, 1024), (-1, 1)):
            x, y = doubles(rng, n, lo, hi), doubles(rng, n, lo, hi)
            q, left = host("div", x, y)
            assert np.array_equal(q.view(np.uint64), (x / y).view(np.uint64))
            assert lo == -1022 or left == 0
        x = doubles(rng, n, -1022, 1024, signed=False)
        r, left = host("sqrt", x)
        assert left == 0 and np.array_equal(r, np.sqrt(x))


FUNS = {
    "sin": lambda r: np.concatenate([r.uniform(-8, 8, 800), doubles(r, 800, -60, 15)]),
    "cos": lambda r: np.concatenate([r.uniform(-8, 8, 800), doubles(r, 800, -60, 15)]),
    "exp": lambda r: np.concatenate([r.uniform(-699, 699, 800), doubles(r, 800, -60, 9)]),
    "log": lambda r: np.concatenate([1 + doubles(r, 800, -52, -1), doubles(r, 800, -1022, 1024,
                                                                          signed=False)]),
    "tanh": lambda r: np.concatenate([r.uniform(-3, 3, 800), doubles(r, 800, -60, 6)]),
}


@pytest.mark.parametrize("name", sorted(FUNS))
def test_functions_are_within_their_error_bound(host, name):
    mp = pytest.importorskip("mpmath")
    mp.mp.prec = 160
    x = FUNS[name](np.random.default_rng(3))
    got, left = host(name, x)
    assert left <= (2 if name in ("sin", "cos") else 0)
    f = getattr(mp, name)
    for g, v in zip(got.tolist(), x.tolist()):
        if g != g:
            continue  # left to CUDA's function
        t = f(mp.mpf(v))
        if t == 0:
            assert g == 0
            continue
        ulp = mp.mpf(2) ** (mp.floor(mp.log(abs(t), 2)) - 52)
        assert abs(mp.mpf(g) - t) <= mp.mpf("0.6") * ulp, (name, v, g)


def _tape(op, binary):
    return S.Tape([C.OP_INPUT, C.OP_INPUT, op, C.OP_OUTPUT], [0, 1, 2, 0], [0, 1, 0, 2],
                  [0, 0, 1 if binary else 0, 0], [0.0] * 4, [1, 1], [1], 3)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["div", "sqrt"] + sorted(FUNS))
def test_the_gpu_gives_the_host_compilation_s_bits(gpu_lib, host, name):
    """Every routine on the GPU against the host compilation: the same bits (log and tanh, whose
    reciprocal starts from the GPU's single-precision seed: within one ulp), CUDA's functions on
    zeros, subnormals, infinities and NaN, at instance counts around a tile."""
    import torch

    from casadi_gb300.runtime import CudaTape
    op = {"div": C.OP_DIV, "sqrt": C.OP_SQRT, "sin": C.OP_SIN, "cos": C.OP_COS, "exp": C.OP_EXP,
          "log": C.OP_LOG, "tanh": C.OP_TANH}[name]
    rng = np.random.default_rng(5)
    tape = CudaTape(_tape(op, name == "div"))
    npf = {"div": np.divide}.get(name) or getattr(np, name)
    for n in (1, 31, 33, 5000):
        if name in FUNS:
            x = FUNS[name](rng)[rng.integers(0, 1600, n)]
        else:
            x = doubles(rng, n, -1022, 1024, signed=name == "div")
        y = doubles(rng, n, -1022, 1024)
        if n > 100:
            x[:SPECIAL.size ** 2] = np.repeat(SPECIAL, SPECIAL.size)
            y[:SPECIAL.size ** 2] = np.tile(SPECIAL, SPECIAL.size)
        got = tape.eval([torch.from_numpy(v[None].copy()).cuda() for v in (x, y)])[0][0].cpu().numpy()
        with np.errstate(all="ignore"):
            want, _ = host(name, x, y) if name == "div" else host(name, x)
            lib = npf(x, y) if name == "div" else npf(x)
        if name in ("div", "sqrt"):
            ok = np.isnan(lib) & np.isnan(got) | (got.view(np.uint64) == lib.view(np.uint64))
        else:
            with np.errstate(all="ignore"):
                close = np.abs(got - lib) <= 2 * np.spacing(np.abs(lib))
                near = np.abs(got - want) <= (
                    np.spacing(np.abs(want)) if name in ("log", "tanh") else 0)
            ok = np.where(np.isnan(want), (got == lib) | close | np.isnan(lib) & np.isnan(got), near)
        assert ok.all(), (name, n, x[~ok][:4], y[~ok][:4], got[~ok][:4])
