"""Persistent multi-tape batches (casadi_gb300_batch_*): several tapes over their own
instance ranges in one launch must give the same numbers as evaluating each tape on its own
(the per-tape value sweep and the per-tape adjoint sweep run the same device arithmetic, so
the comparison is bit for bit), and the oracle's within the documented tolerance."""
import numpy as np
import pytest

import oracle as O
from casadi_gb300 import runtime as R
from casadi_gb300 import workloads as W

from helpers import RTOL, assert_close, magnitudes, same_bits, value_bounds

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _items():
    """(Function, n, nadj, inputs) covering eval-only and adjoint items, ragged tiles, a
    one-instance item, two tapes of very different length, and split items (two or more
    directions) recorded cooperatively before the launch (few tiles) or by record units."""
    out = []
    f = W.cartpole_rollout(4)
    out.append((f, 1000, 1, W.cartpole_inputs(1000, steps=4, seed=1)))
    out.append((f, 33, 2, W.cartpole_inputs(33, steps=4, seed=2)))
    # two directions over more tiles than the cooperative pre-record takes: per-tile record
    # units inside the persistent launch
    out.append((f, 20000, 2, W.cartpole_inputs(20000, steps=4, seed=7)))
    g = W.random_dag(n_in=16, n_nodes=3000, n_out=4, seed=3, window=64, bounded=True)
    out.append((g, 5000, 1, W.dag_inputs(5000, n_in=16, seed=3)))
    out.append((g, 1, 0, W.dag_inputs(1, n_in=16, seed=4)))
    h = W.random_dag(n_in=16, n_nodes=300, n_out=4, seed=5, window=32, bounded=True)
    out.append((h, 777, 0, W.dag_inputs(777, n_in=16, seed=5)))
    out.append((h, 64, 3, W.dag_inputs(64, n_in=16, seed=6)))
    return out


def _seeds(f, n, nadj, seed):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal((nadj, k, n)) for k in f.tape.nnz_out]


@pytest.mark.parametrize("graph", [False, True])
def test_batch_matches_per_tape_sweeps(gpu_lib, graph):
    items = _items()
    tapes = {}
    b = R.Batch()
    queued = []
    for k, (f, n, nadj, args) in enumerate(items):
        t = tapes.setdefault(id(f), R.CudaTape(f))
        dargs = [_cuda(a) for a in args]
        dseeds = [_cuda(s) for s in _seeds(f, n, nadj, k)] if nadj else None
        res, asens = b.add(t, dargs, dseeds)
        queued.append((t, dargs, dseeds, res, asens))
    b.run(graph=graph)
    if graph:
        b.run(graph=True)  # replay
    b.status()
    for t, dargs, dseeds, res, asens in queued:
        t.sync()
        if dseeds is None:
            want = t.eval(dargs)
            for g, w in zip(res, want):
                assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all()
        else:
            want_r, want_s = t.reverse(dargs, dseeds)
            for g, w in zip(res, want_r):
                assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all()
            for g, w in zip(asens, want_s):
                assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all()


def test_batch_matches_oracle(gpu_lib):
    items = _items()
    b = R.Batch()
    queued = []
    for k, (f, n, nadj, args) in enumerate(items):
        t = R.CudaTape(f)
        seeds = _seeds(f, n, nadj, k) if nadj else None
        res, asens = b.add(t, [_cuda(a) for a in args],
                           [_cuda(s) for s in seeds] if seeds else None)
        queued.append((f, n, args, seeds, res, asens, t))
    b.run()
    b.status()
    for k, (f, n, args, seeds, res, asens, t) in enumerate(queued):
        t.sync()
        # thousands of sin/cos/exp/tanh nodes carry the <= 1-ulp differences between CUDA's and
        # the host libm into values and adjoints: element-wise bounds from the oracle
        want = O.eval(f.tape, args, n)
        vb = value_bounds(f.tape, args, n)
        for j, (g, w) in enumerate(zip(res, want)):
            assert_close(g.cpu().numpy(), w, "item %d value %d" % (k, j), bound=vb[j])
        if seeds:
            for d in range(seeds[0].shape[0]):
                sd = [s[d:d + 1] for s in seeds]
                _, ws = O.reverse(f.tape, args, sd, n)
                _, ms = magnitudes(O.reverse, f.tape, args, sd, n)
                for j, (w, m) in enumerate(zip(ws, ms)):
                    assert_close(asens[j][d].cpu().numpy(), w[0],
                                 "item %d adjoint %d/%d" % (k, d, j), bound=RTOL * m[0])


def test_batch_graph_replay_sees_new_inputs(gpu_lib):
    """A replayed graph reads the inputs' current contents (same pointers, new values)."""
    f = W.cartpole_rollout(4)
    t = R.CudaTape(f)
    n = 300
    args = [_cuda(a) for a in W.cartpole_inputs(n, steps=4, seed=11)]
    seeds = [_cuda(s) for s in _seeds(f, n, 1, 11)]
    b = R.Batch()
    res, asens = b.add(t, args, seeds)
    b.run(graph=True)
    new = W.cartpole_inputs(n, steps=4, seed=12)
    for a, v in zip(args, new):
        a.copy_(_cuda(v))
    b.run(graph=True)
    want_r, want_s = t.reverse(args, seeds)
    for g, w in zip(res + asens, want_r + want_s):
        assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all()


def test_batch_rejects_small_scratch_and_bad_ids(gpu_lib):
    import ctypes as ct
    lib = R.load()
    assert lib.casadi_gb300_batch_run(12345, None, 0, 0, None) == -1
    f = W.cartpole_rollout(2)
    t = R.CudaTape(f)
    b = R.Batch()
    args = [_cuda(a) for a in W.cartpole_inputs(64, steps=2, seed=1)]
    b.add(t, args, [_cuda(s) for s in _seeds(f, 64, 1, 1)])
    assert b.scratch_bytes() > 0
    st = lib.casadi_gb300_batch_run(b.id, None, 0, 0, ct.c_void_p(0))
    assert st == -5
    assert lib.casadi_gb300_batch_add(b.id, 999999, 1, 1, 0, None, None, None, None) == -1


@pytest.mark.parametrize("mode", [1, 2])
def test_batch_residence_gives_the_same_bits(gpu_lib, mode):
    """The batch with its work vectors forced into global (1) or shared (2) memory."""
    items = _items()
    tapes = {}
    b = R.Batch()
    b.set_residence(mode)
    queued = []
    for k, (f, n, nadj, args) in enumerate(items):
        t = tapes.setdefault(id(f), R.CudaTape(f))
        dargs = [_cuda(a) for a in args]
        dseeds = [_cuda(s) for s in _seeds(f, n, nadj, k)] if nadj else None
        res, asens = b.add(t, dargs, dseeds)
        queued.append((t, dargs, dseeds, res, asens))
    b.run(graph=True)
    b.status()
    for t, dargs, dseeds, res, asens in queued:
        if dseeds is None:
            for g, w in zip(res, t.eval(dargs)):
                assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all()
        else:
            want_r, want_s = t.reverse(dargs, dseeds)
            for g, w in zip(res + asens, want_r + want_s):
                assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all()


@pytest.mark.parametrize("others", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 33, 1000, 40000])
def test_one_colour_jacobians_in_a_batch_of_teams(gpu_lib, n, others):
    """A coloured Jacobian of one colour has one direction and is not split, unlike one of more
    colours: alone and beside value, adjoint and two-colour items, on a tape whose work vector leaves
    few warps per SM (the batch by teams) and on a narrow one, the general forward sweep's bits."""
    wide = W.random_dag(n_in=20, n_nodes=900, n_out=5, seed=4, window=256, bounded=True)
    narrow = W.random_dag(n_in=20, n_nodes=200, n_out=3, seed=5, window=16, bounded=True)
    tapes = [R.CudaTape(f) for f in (wide, narrow)]
    assert tapes[0].sz_w >= 60  # fewer than 20 one-warp CTAs of the record sweep fit an SM
    args = [_cuda(a) for a in W.dag_inputs(n, n_in=20, seed=6)]
    b = R.Batch()
    queued, checks = [], []
    for t, f in zip(tapes, (wide, narrow)):
        color = np.full(20, -1, np.int32)
        color[::3] = 0
        seeds = torch.zeros((1, 20, n), dtype=torch.float64, device="cuda")
        seeds[0, ::3] = 1.0
        queued.append((b.add_jacobian_colored(t, args, 1, color), t, seeds))
        if others:
            aseeds = [_cuda(s) for s in _seeds(f, n, 1, 7)]
            checks.append((b.add(t, args, aseeds), t, aseeds))
        if others > 1:
            two = np.arange(20, dtype=np.int32) % 2
            seeds = torch.stack([_cuda(np.repeat((two == d)[:, None] * 1.0, n, 1)) for d in (0, 1)])
            queued.append((b.add_jacobian_colored(t, args, 2, two), t, seeds))
    for graph in (False, True, True):
        for comp, _, _ in queued:
            for c in comp:
                c.fill_(float("nan"))
        b.run(graph=graph)
        b.status()
        for comp, t, seeds in queued:
            _, want = t.forward(args, [seeds])
            for g, w in zip(comp, want):
                assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all()
        for (res, asens), t, aseeds in checks:
            want_r, want_s = t.reverse(args, aseeds)
            for g, w in zip(res + asens, want_r + want_s):
                assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all()


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("nadj", [0, 1, 3])
def test_batch_whose_tape_was_freed_is_refused(gpu_lib, nadj, graph):
    """Whole items and split ones (three directions: recorded by a launch of their own): after the
    tape is freed a run is refused before anything is launched, prepared or captured before or not,
    and the batch's other results stay as they were."""
    lib = R.load()
    f = W.cartpole_rollout(4)
    args = [_cuda(a) for a in W.cartpole_inputs(200, steps=4, seed=3)]
    for prepared in (False, True):
        t = R.CudaTape(f)
        b = R.Batch()
        res, _ = b.add(t, args, [_cuda(s) for s in _seeds(f, 200, nadj, 3)] if nadj else None)
        if prepared:
            b.run(graph=graph)
            b.status()
        before = [r.clone() for r in res]
        assert lib.casadi_gb300_tape_free(t.id) == 0
        with pytest.raises(R.CasadiGpuError, match="is gone"):
            b.run(graph=graph)
        torch.cuda.synchronize()
        if prepared:
            for g, w in zip(res, before):
                assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all()
        t.id = None


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_small_operations_in_a_persistent_batch(gpu_lib, mode):
    """Comparisons, logic, minima, selections, signs and rounding have cases of their own in the
    persistent batch: values and adjoints on zeros, infinities, NaN and ordinary arguments, the bits of
    the sweeps of one tape (which call them)."""
    from casadi_gb300 import calculus as C
    from casadi_gb300 import sx as S
    rng = np.random.default_rng(2)
    v = np.concatenate([[0.0, -0.0, np.inf, -np.inf, np.nan, 1.0, -1.0, 0.5, -2.5, 5e-324, -1e300],
                        rng.standard_normal(6)])
    args = [_cuda(w.ravel()[None]) for w in np.meshgrid(v, v)]
    n = v.size ** 2
    seed = _cuda(rng.standard_normal((1, 1, n)))
    b = R.Batch()
    b.set_residence(mode)
    queued = []
    for op in (C.OP_LT, C.OP_LE, C.OP_EQ, C.OP_NE, C.OP_NOT, C.OP_AND, C.OP_OR, C.OP_FLOOR, C.OP_CEIL,
               C.OP_SIGN, C.OP_COPYSIGN, C.OP_IF_ELSE_ZERO, C.OP_FMIN, C.OP_FMAX):
        two = op in C.BINARY_OPS
        t = R.CudaTape(S.Tape([C.OP_INPUT, C.OP_INPUT, op, C.OP_OUTPUT], [0, 1, 2, 0], [0, 1, 0, 2],
                              [0, 0, 1 if two else 0, 0], [0.0] * 4, [1, 1], [1], 3))
        queued.append((op, t, b.add(t, args)[0], []))
        queued.append((op, t) + tuple(b.add(t, args, [seed])))
    b.run()
    b.status()
    for op, t, res, asens in queued:
        want_r, want_s = t.reverse(args, [seed])
        for g, w in zip(list(res) + list(asens), list(want_r) + list(want_s if asens else [])):
            assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all(), C.OP_NAMES[op]


@pytest.mark.parametrize("units", [0, 1, 7 * 152 + 3])
@pytest.mark.parametrize("nadj", [0, 1, 2])
def test_batches_on_both_sides_of_a_full_gpu(gpu_lib, nadj, units):
    """Batches of as many units as are resident at 20 one-warp CTAs per SM, one more and some more (the
    form of fewer registers): the bits of the sweeps of one tape."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    f = W.cartpole_rollout(1)
    t = R.CudaTape(f)
    assert t.sz_w <= 30  # registers, not shared memory, decide how many CTAs are resident
    n = 32 * ((20 * sms + units) // max(1, nadj)) - 3  # a unit per tile, or per tile and direction
    args = [_cuda(a) for a in W.cartpole_inputs(n, steps=1, seed=units)]
    seeds = [_cuda(s) for s in _seeds(f, n, nadj, 9)] if nadj else None
    b = R.Batch()
    res, asens = b.add(t, args, seeds)
    b.run()
    b.status()
    want_r, want_s = t.reverse(args, seeds) if nadj else (t.eval(args), [])
    for g, w in zip(list(res) + list(asens), list(want_r) + list(want_s)):
        assert same_bits(g.cpu().numpy(), w.cpu().numpy()).all()


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("slots", [905, 906, 907, 908])
def test_batch_at_the_shared_memory_limit(gpu_lib, slots, mode):
    """Work vectors of up to 908 slots (227 KB) run in a batch whether or not the entry ring has room
    beside them, with the bits of the sweeps of one tape."""
    from casadi_gb300 import sx as S
    k, n = 2 * (slots - 5), 65
    x = S.sym("x", k)
    p = [x[i] * x[(i + 1) % k] for i in range(k)]
    q = [p[i] + p[k - 1 - i] for i in range(k // 2)]
    prod = q[0]
    for v in q[1:]:
        prod = prod * v
    t = R.CudaTape(S.Function("w", [x], [[prod, sum(p[1:], p[0])]]))
    assert t.sz_w == slots
    g = torch.Generator(device="cuda").manual_seed(slots)
    args = [torch.rand((k, n), dtype=torch.float64, device="cuda", generator=g) * 1e-3 + 0.7]
    seeds = [torch.rand((1, 2, n), dtype=torch.float64, device="cuda", generator=g)]
    b = R.Batch()
    b.set_residence(mode)
    res, asens = b.add(t, args, seeds)
    values, _ = b.add(t, args)
    b.run()
    b.status()
    want_r, want_s = t.reverse(args, seeds)
    for got, w in zip(list(res) + list(asens) + list(values), list(want_r) + list(want_s) + list(want_r)):
        assert same_bits(got.cpu().numpy(), w.cpu().numpy()).all()
