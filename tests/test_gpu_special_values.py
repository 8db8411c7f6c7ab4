"""Zeros, infinities, NaN, subnormals and results at the ends of the exponent range, in warps
that mix them with ordinary arguments."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

VALUES = [0.0, -0.0, 1.0, -1.0, 0.3, -7.25, 1e5, -3e9, 1e300, -1e308, np.inf, -np.inf, np.nan, 5e-324,
          -5e-324, 3e-310, 2.2250738585072014e-308, 709.0, 709.8, 745.9, 746.0, -708.5, -745.0, -745.2,
          -746.0, 1e-200, 40.0, -40.0]
OPS = {"div": np.divide, "sqrt": np.sqrt, "sin": np.sin, "cos": np.cos, "exp": np.exp, "log": np.log,
       "tanh": np.tanh}


@pytest.mark.parametrize("residence", [2, 3])
@pytest.mark.parametrize("op", sorted(OPS))
def test_special_values(gpu_lib, op, residence):
    """Against numpy: infinities, zeros with their signs and NaN alike, finite results within two
    units in the last place (numpy's functions and these are each within one)."""
    import torch
    from casadi_gb300 import runtime as R, sx as S
    x = S.sym("x", 2)
    expr = x[0] / x[1] if op == "div" else getattr(S, op)(x[0])
    ct = R.CudaTape(S.Function("f", [x], [[expr]]))
    ct.set_residence(residence)
    a, b = (v.ravel() for v in np.meshgrid(VALUES, VALUES))
    got, = ct.eval([torch.from_numpy(np.stack([a, b])).cuda()])
    got = got.cpu().numpy()[0]
    with np.errstate(all="ignore"):
        want = OPS[op](a, b) if op == "div" else OPS[op](a)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    ok = ~np.isnan(want)
    special = ok & (np.isinf(want) | (want == 0))
    assert np.array_equal(got[special], want[special])
    assert np.array_equal(np.signbit(got[special]), np.signbit(want[special]))
    fin = ok & ~special
    assert np.all(np.abs(got[fin] - want[fin]) <= 2 * np.spacing(np.abs(want[fin])))
    ct.sync()
