"""Constant operands in the derivative sweeps: their partials are not stored, no adjoint goes to
them, and the factor of a product with a constant (the reciprocal of a constant divisor) comes
from the tape's table instead of the recorded partials. Every op with a constant in either place,
constants shared and in both places, against the oracle, in every variant."""
import numpy as np
import pytest

import oracle as O
from casadi_gb300 import runtime as R
from casadi_gb300 import sx as S

from helpers import assert_bitexact

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _dev(arrs):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrs]


def _host(ts):
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in ts]


def _function():
    x = S.sym("x", 4)
    c = 0.3
    a = [c * x[0], x[1] * c, x[2] / 3.0, 2.5 / (x[3] + 3.0), c + x[0], x[1] - c, c - x[2],
         S.fmin(x[0], 0.25), S.fmax(0.25, x[1]), S.if_else_zero(S.lt(x[2], c), 1.5 * x[3]),
         S.copysign(x[0], -1.0)]
    b = [a[0] * a[1] + 0.7 * a[2], a[3] * (0.7 * a[3]), (a[4] * a[5]) / 3.0 - a[6],
         a[7] * a[8] * 0.3, a[9] + a[10] * 0.1]
    return S.Function("K", [x], [[b[0] * b[1], b[2] - 0.5 * b[3], b[4] * b[0]], [S.const(0.3)]])


@pytest.mark.parametrize("n", [1, 33, 3000])
def test_constant_operands_in_every_variant(gpu_lib, n):
    f = _function()
    t = f.tape
    rng = np.random.default_rng(n)
    args = [rng.uniform(-1, 1, (4, n))]
    fseeds = [rng.standard_normal((5, 4, n))]
    aseeds = [rng.standard_normal((2, 3, n)), rng.standard_normal((2, 1, n))]
    _, wf = O.forward(t, args, fseeds, n)
    _, wj = O.jacobian(t, args, n)
    _, wa = O.reverse(t, args, aseeds, n)
    ct = R.CudaTape(f)
    for v in [-1] + list(range(R.TAN_WINDOWED + 1)):
        ct.set_variant(0, v)
        ct.set_variant(1, v)
        ct.set_variant(2, min(v, R.N_ADJ_VARIANTS - 1))
        for got, want, what in ((ct.forward(_dev(args), _dev(fseeds))[1], wf, "forward"),
                                (ct.jacobian(_dev(args))[1], wj, "jacobian"),
                                (ct.reverse(_dev(args), _dev(aseeds))[1], wa, "reverse")):
            for g, w in zip(_host(got), want):
                assert_bitexact(g, w, "%s, variant %d" % (what, v))
    b = R.Batch()
    _, asens = b.add(ct, _dev(args), _dev(aseeds))
    b.run()
    b.status()
    for g, w in zip(_host(asens), wa):
        assert_bitexact(g, w, "batch")
    ct.sync()


@pytest.mark.parametrize("factor", [0.5, 4.0, 2.0 ** -1000, 2.0 ** 1000, 2.0 ** -1022, -0.5])
def test_tangents_of_products_with_powers_of_two(gpu_lib, factor):
    """A product's tangent with a power of two as the partial is an exponent addition: seeds that
    are zero, subnormal, huge, infinite or NaN, and results that leave the normal range, in every
    variant, against the oracle's product."""
    x = S.sym("x", 2)
    t = S.Function("P", [x], [[factor * x[0], x[1] * factor + 0.25 * x[0]]]).tape
    v = np.array([0.0, -0.0, 1.0, -3.7, 1e-300, -1e300, 5e-324, 2.2250738585072014e-308, np.inf, -np.inf,
                  np.nan, 1.7976931348623157e308, 3e-310, 2.0 ** -50, 1e154])
    seeds = np.stack([v, v[::-1]])[None]
    seeds = np.concatenate([np.tile(seeds, (1, 1, 9)), np.ones((1, 2, 135))])
    n = seeds.shape[2]
    args = [np.random.default_rng(1).standard_normal((2, n))]
    with np.errstate(all="ignore"):
        _, want = O.forward(t, args, [seeds], n)
        _, wj = O.jacobian(t, args, n)
    ct = R.CudaTape(t)
    for k in range(R.TAN_WINDOWED + 1):
        ct.set_variant(0, k)
        ct.set_variant(1, k)
        for g, w in zip(_host(ct.forward(_dev(args), _dev([seeds]))[1]), want):
            assert_bitexact(g, w, "forward, variant %d" % k)
        for g, w in zip(_host(ct.jacobian(_dev(args))[1]), wj):
            assert_bitexact(g, w, "jacobian, variant %d" % k)
    ct.sync()
