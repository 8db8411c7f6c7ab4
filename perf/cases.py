"""Performance cases of the GB300 SX-tape evaluator: what a user's program has it do, through
its public entry points, with the sizes of the repository's own workloads and benchmark.

A case names a ``kind`` (which entry point on which family of tapes) and its sizes. Tapes,
colourings and other handles are built once per shape and kept, as a program that evaluates
many batches of inputs keeps them; inputs are drawn on the device from the seed alone, with the
distributions of the workloads.
"""
import functools
import math

import numpy as np
import torch

DEV = "cuda"
F64 = torch.float64

# FP64 operations per instance, libm calls at their measured cost in FP64 instructions: the
# cart-pole RK4 step (values, values with partials, one adjoint direction), one tangent
# direction through one step, and per node of the bounded random DAG.
STEP_EVAL, STEP_RECORD, STEP_ADJ, STEP_TAN = 318, 466, 185, 129
NODE_EVAL, NODE_RECORD, NODE_ADJ, NODE_INSTR = 8.5, 10.7, 1.9, 1.37
QUAD_RECORD, QUAD_GRAD, QUAD_DIR = 2200, 4800, 1500  # quadcopter, per interval

LISTED = [
    # the smallest call: one controller's worth of plant steps, where launches and latency count
    dict(name="step_small", kind="eval", tape="step", n=100),
    # the cart-pole step over 65536 instances, values only (sampling and simulation)
    dict(name="step", kind="eval", tape="step", n=65536),
    # Jacobian of xN and gradient of the cost of a 20-step rollout for about a thousand
    # starting points (a trajectory optimiser's multi-start), an odd count
    dict(name="sensitivities_small", kind="jacrev", steps=20, n=1001),
    # the same over 262144 instances: the benchmark's step
    dict(name="sensitivities", kind="jacrev", steps=20, n=262144),
    # the same from page-locked host buffers in CasADi's Map layout, copies included
    dict(name="host_map", kind="host", steps=20, n=65536),
    # directional derivatives: five general forward seeds through the rollout
    dict(name="forward", kind="forward", steps=20, nfwd=5, n=50001),
    # a general expression graph of 10000 nodes: values and the adjoint of its outputs
    dict(name="dag_adjoint", kind="dag_adjoint", nodes=10000, n=16384),
    # bit-vector sparsity propagation through the same graph, both ways
    dict(name="dag_sparsity", kind="dag_sparsity", nodes=10000, n=16384),
    # a mixed queue: eight graphs of 200 to 20000 nodes, log-normal instance counts, values and
    # adjoints in one persistent launch
    dict(name="mixed_batch", kind="batch", total=1 << 18),
    # scenario MPC: sparse constraint Jacobian and Lagrangian Hessian of a multiple-shooting
    # quadcopter problem over 4096 scenarios, in one graph launch
    dict(name="mpc_kkt", kind="kkt", intervals=100, n=4096, graph=True),
    # gradient of a cost summed over scenarios with respect to shared controls (MapSum)
    dict(name="summed_cost", kind="mapsum", steps=20, n=131072),
    # 100-step rollout differentiated through torch.autograd, checkpointed every 10 steps
    dict(name="autograd_rollout", kind="autograd", steps=100, n=131072),
]


def listed():
    return [dict(c) for c in LISTED]


def _log(rng, lo, hi):
    return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["eval", "jacrev", "host", "forward", "dag_adjoint", "dag_sparsity",
                       "batch", "kkt", "mapsum", "autograd"])
    if kind == "eval":
        tape = rng.choice(["step", "rollout"])
        return dict(kind=kind, tape=tape, n=_log(rng, 1, 65536 if tape == "step" else 262144))
    if kind == "jacrev":
        return dict(kind=kind, steps=rng.randint(5, 20), n=_log(rng, 50, 262144))
    if kind == "host":
        return dict(kind=kind, steps=rng.randint(5, 20), n=_log(rng, 500, 65536))
    if kind == "forward":
        return dict(kind=kind, steps=rng.randint(5, 20), nfwd=rng.randint(1, 8),
                    n=_log(rng, 200, 100000))
    if kind in ("dag_adjoint", "dag_sparsity"):
        return dict(kind=kind, nodes=_log(rng, 200, 10000), n=_log(rng, 300, 16384))
    if kind == "batch":
        return dict(kind=kind, total=_log(rng, 4096, 1 << 18))
    if kind == "kkt":
        return dict(kind=kind, intervals=rng.randint(5, 30), n=_log(rng, 64, 4096),
                    graph=rng.random() < 0.5)
    if kind == "mapsum":
        return dict(kind=kind, steps=rng.randint(5, 20), n=_log(rng, 500, 131072))
    return dict(kind=kind, steps=10 * rng.randint(2, 10), n=_log(rng, 1000, 131072))


# ---- handles a program builds once ------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _cartpole(steps):
    """The RK4 step (steps = 0) or a rollout, as a registered tape."""
    from casadi_gb300 import workloads as W
    from casadi_gb300.runtime import CudaTape
    return CudaTape(W.cartpole_rollout(steps) if steps else W.cartpole_step())


DAG_IN, DAG_OUT, DAG_WINDOW = 64, 16, 256
DAG_P = [0.25, 0.15, 0.25, 0.05, 0.06, 0.06, 0.06, 0.04, 0.04, 0.04]


@functools.lru_cache(maxsize=None)
def _dag_nodes(nodes, seed):
    """A random graph's node list: op codes (add, sub, mul, div, sin, cos, exp, log, sqrt,
    tanh) and two operands each, drawn from the previous 256 nodes."""
    rng = np.random.default_rng(seed)
    k = np.arange(DAG_IN, nodes)
    op = rng.choice(10, size=k.size, p=DAG_P)
    lo = np.maximum(0, k - DAG_WINDOW)
    return op, rng.integers(lo, k), rng.integers(lo, k)


@functools.lru_cache(maxsize=None)
def _dag(nodes, seed):
    from casadi_gb300 import workloads as W
    from casadi_gb300.runtime import CudaTape
    op, a, b = _dag_nodes(nodes, seed)
    return CudaTape(W.dag_from_nodes(DAG_IN, DAG_OUT, op, a, b, bounded=True))


@functools.lru_cache(maxsize=None)
def _kkt(intervals):
    from casadi_gb300 import sparse_ad, workloads as W
    w, x0bar, obj, g = W.quad_ms_nlp(intervals)
    return sparse_ad.KKT(w, x0bar, obj, g)


@functools.lru_cache(maxsize=None)
def _autograd(steps):
    from casadi_gb300.autograd import CheckpointedRollout
    return CheckpointedRollout(steps, 10)


def _mixed_items(total):
    """(graph, instances) of a mixed queue: eight graphs of 200..20000 nodes, log-normal
    counts of median 4096 (scaled down for short queues), at most 24 items."""
    rng = np.random.default_rng(7)
    nodes = np.exp(np.linspace(math.log(200), math.log(20000), 8)).astype(int)
    median = min(4096, max(64, total // 16))
    items, left = [], total
    while left > 0:
        n = left if len(items) == 23 else int(min(left, max(1, rng.lognormal(math.log(median), 1.5))))
        items.append((int(nodes[int(rng.integers(8))]), n))
        left -= n
    return items


# ---- inputs -------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _uniform(g, lo, hi, rows, n):
    return torch.rand((rows, n), generator=g, device=DEV, dtype=F64) * (hi - lo) + lo


def _cartpole_inputs(g, n, steps):
    hi = torch.tensor([[2.0], [3.0], [math.pi], [5.0]], device=DEV, dtype=F64)
    return [_uniform(g, -1.0, 1.0, 4, n) * hi, _uniform(g, -10.0, 10.0, max(1, steps), n)]


def _dag_inputs(g, n):
    return torch.randn((DAG_IN, n), generator=g, device=DEV, dtype=F64)


def _kkt_inputs(g, n, K):
    state = torch.tensor([1.0] * 3 + [0.5] * 9, device=DEV, dtype=F64)
    one = torch.cat([state, torch.tensor([1.0, 0.05, 0.05, 0.05], device=DEV, dtype=F64)])
    scale = torch.cat([one.repeat(K), state])[:, None]
    w = _uniform(g, -1.0, 1.0, 16 * K + 12, n) * scale
    w[12:16 * K:16] += 9.81
    x0 = _uniform(g, -1.0, 1.0, 12, n)
    x0[3:6] = 0.0
    x0[9:12] = 0.0
    x0[6:9] *= 0.5
    lam = torch.randn((12 * (K + 1), n), generator=g, device=DEV, dtype=F64)
    return [w, x0, torch.ones((1, n), device=DEV, dtype=F64), lam]


def _rand_bits(g, rows, n):
    return torch.randint(-2**63, 2**63 - 1, (rows, n), generator=g, device=DEV, dtype=torch.int64)


def _cost_seed(n, lead=1):
    return [torch.zeros((lead, 4, n), device=DEV, dtype=F64),
            torch.ones((lead, 1, n), device=DEV, dtype=F64)]


def _pinned(t):
    """A device tensor (nnz, n) as CasADi's page-locked instance-major host array (n, nnz)."""
    h = torch.empty((t.shape[1], t.shape[0]), dtype=F64, pin_memory=True)
    h.copy_(t.T)
    return h.numpy()


def _pinned_empty(*shape):
    return torch.empty(shape, dtype=F64, pin_memory=True).numpy()


def _inputs(case, seed):
    """The device inputs of a case, from the seed alone."""
    g, kind = _gen(seed), case["kind"]
    if kind == "eval":
        return _cartpole_inputs(g, case["n"], 20 if case["tape"] == "rollout" else 1)
    if kind in ("jacrev", "host", "autograd"):
        return _cartpole_inputs(g, case["n"], case["steps"])
    if kind == "forward":
        args = _cartpole_inputs(g, case["n"], case["steps"])
        shape = (case["nfwd"], 4 + case["steps"], case["n"])
        s = torch.randn(shape, generator=g, device=DEV, dtype=F64)
        return args + [s[:, :4].contiguous(), s[:, 4:].contiguous()]
    if kind == "mapsum":
        x0, u = _cartpole_inputs(g, case["n"], case["steps"])
        return [x0, u[:, 0].contiguous()]
    if kind == "dag_adjoint":
        return [_dag_inputs(g, case["n"]),
                torch.ones((1, DAG_OUT, case["n"]), device=DEV, dtype=F64)]
    if kind == "dag_sparsity":
        return [_rand_bits(g, DAG_IN, case["n"]), _rand_bits(g, DAG_OUT, case["n"])]
    if kind == "batch":
        return [_dag_inputs(g, n) for _, n in _mixed_items(case["total"])]
    return _kkt_inputs(g, case["n"], case["intervals"])


def prepare(case, seed):
    kind, x = case["kind"], _inputs(case, seed)
    n = case.get("n")
    s = {"kind": kind, "x": x}
    if kind == "eval":
        s["f"] = _cartpole(20 if case["tape"] == "rollout" else 0)
    elif kind == "jacrev":
        s["f"] = _cartpole(case["steps"])
        s["seeds"] = _cost_seed(n)
        nz = 4 + case["steps"]
        # the Jacobian of xN alone: the cost's row is the adjoint's result
        s["jac"] = [torch.empty((nz, 4, n), dtype=F64, device=DEV), None]
    elif kind == "host":
        from casadi_gb300.runtime import CudaMap
        nz = 4 + case["steps"]
        s["f"] = CudaMap(_cartpole(case["steps"]), n)
        s["x"] = [_pinned(t) for t in x]
        s["seeds"] = [_pinned(t[0]).reshape(n, 1, -1) for t in _cost_seed(n)]
        s["res"] = [_pinned_empty(n, 4), _pinned_empty(n, 1)]
        s["jac"] = [_pinned_empty(n, nz, 4), None]
        s["asens"] = [_pinned_empty(n, 1, 4), _pinned_empty(n, 1, case["steps"])]
    elif kind == "forward":
        s["f"] = _cartpole(case["steps"])
    elif kind in ("dag_adjoint", "dag_sparsity"):
        s["f"] = _dag(case["nodes"], 0)
    elif kind == "batch":
        from casadi_gb300.runtime import Batch
        s["f"], s["out"] = Batch(), []
        for (nodes, m), a in zip(_mixed_items(case["total"]), x):
            seeds = torch.ones((1, DAG_OUT, m), dtype=F64, device=DEV)
            s["out"].append(s["f"].add(_dag(nodes, 0), [a], [seeds]))
    elif kind == "kkt":
        s["f"] = _kkt(case["intervals"])
        if case["graph"]:
            s["run"] = s["f"].batched(x)
    elif kind == "mapsum":
        from casadi_gb300.runtime import CudaMapSum
        s["f"] = CudaMapSum(_cartpole(case["steps"]), n, [False, True], [False, True])
        s["seeds"] = [torch.zeros((1, 4, n), dtype=F64, device=DEV),
                      torch.ones((1, 1), dtype=F64, device=DEV)]
    else:
        s["f"] = _autograd(case["steps"])
        for t in x:
            t.requires_grad_(True)
    return s


def run(s):
    kind, f, x = s["kind"], s["f"], s["x"]
    if kind == "eval":
        return f.eval(x)
    if kind == "jacrev":
        return f.jacobian_reverse(x, s["seeds"], jac=s["jac"])
    if kind == "host":
        return f.jacobian_reverse(x, s["seeds"], res=s["res"], jac=s["jac"], asens=s["asens"])
    if kind == "forward":
        return f.forward(x[:2], x[2:])
    if kind == "dag_adjoint":
        return f.reverse(x[:1], x[1:])
    if kind == "dag_sparsity":
        fwd = f.sp_forward(x[:1])
        seeds = x[1].clone()  # consumed by the reverse sweep
        back = torch.zeros_like(x[0])
        f.sp_reverse([back], [seeds])
        return fwd, back
    if kind == "batch":
        f.run(graph=True)
        return s["out"]
    if kind == "kkt":
        return s["run"]() if "run" in s else f(x)
    if kind == "mapsum":
        return f.reverse(x, s["seeds"])
    for t in x:
        t.grad = None
    xn, cost = f(x[0], x[1])
    cost.sum().backward()
    return xn.detach(), cost.detach(), x[0].grad, x[1].grad


def work(case):
    kind, n, S = case["kind"], case.get("n"), case.get("steps", 20)
    io = 8.0
    if kind == "eval":
        k = 20 if case["tape"] == "rollout" else 1
        return {"bytes": io * n * (4 + k + 4 + (k > 1)), "flops": n * k * STEP_EVAL}
    pairs = 4 * S + S * (S + 1) / 2  # (direction, step) pairs with a nonzero derivative
    if kind in ("jacrev", "host"):
        rows = (4 + S) + 5 + 4 * (4 + S) + 5 + (4 + S)
        return {"bytes": io * n * rows,
                "flops": n * (S * (STEP_RECORD + STEP_ADJ) + pairs * STEP_TAN)}
    if kind == "forward":
        d = case["nfwd"]
        return {"bytes": io * n * ((4 + S + 5) * (1 + d)),
                "flops": n * S * (STEP_RECORD + d * 1.4 * STEP_TAN)}
    if kind == "mapsum":
        return {"bytes": io * n * (4 + 4 + 4 + 4), "flops": n * S * (STEP_RECORD + STEP_ADJ)}
    if kind == "autograd":
        return {"bytes": io * n * (2 * (4 + S) + 5),
                "flops": n * S * (STEP_EVAL + STEP_RECORD + STEP_ADJ)}
    if kind == "dag_adjoint":
        return {"bytes": io * n * 2 * (DAG_IN + DAG_OUT),
                "flops": n * case["nodes"] * (NODE_RECORD + NODE_ADJ)}
    if kind == "dag_sparsity":
        return {"bytes": io * n * 2 * (DAG_IN + DAG_OUT), "flops": 2.0 * n * case["nodes"] * NODE_INSTR}
    if kind == "batch":
        items = _mixed_items(case["total"])
        return {"bytes": io * case["total"] * 2 * (DAG_IN + DAG_OUT),
                "flops": sum(m * k * (NODE_RECORD + NODE_ADJ) for k, m in items)}
    K = case["intervals"]
    return {"bytes": io * n * (16 * K + 12 * (K + 3) + 118 * K + 110 * K),
            "flops": n * K * (QUAD_RECORD + QUAD_GRAD + 24 * QUAD_DIR)}


# ---- 64-bit values in plain torch ---------------------------------------------------------------
def _ode(x, u):
    mc, mp, l, grav = 1.0, 0.1, 0.5, 9.81
    s, c, om = torch.sin(x[2]), torch.cos(x[2]), x[3]
    den = mc + mp * s * s
    acc = (u + mp * s * (l * om * om + grav * c)) / den
    alpha = (-u * c - mp * l * om * om * c * s - (mc + mp) * grav * s) / (l * den)
    return torch.stack([x[1], acc, om, alpha])


def _rk4(f, x, u, dt):
    k1 = f(x, u)
    k2 = f(x + dt / 2 * k1, u)
    k3 = f(x + dt / 2 * k2, u)
    k4 = f(x + dt * k3, u)
    return x + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)


def _rollout(x, u):
    cost = 0.0
    for k in range(u.shape[0]):
        cost = cost + (x * x).sum(0) + 0.01 * u[k] * u[k]
        x = _rk4(_ode, x, u[k], 0.02)
    return x, cost[None]


def _rows(outs, wrt):
    """Gradients of each output row, summed over instances, with respect to ``wrt``."""
    return [torch.autograd.grad(o.sum(), wrt, retain_graph=True) for o in outs]


def _dag_value(x, nodes, seed):
    op, a, b = _dag_nodes(nodes, seed)
    v = list(x)
    for o, i, j in zip(op.tolist(), a.tolist(), b.tolist()):
        p, q = v[i], v[j]
        v.append(0.5 * (p + q) if o == 0 else 0.5 * (p - q) if o == 1 else
                 p * torch.tanh(q) if o == 2 else p / (q * q + 1.0) if o == 3 else
                 torch.sin(p) if o == 4 else torch.cos(p) if o == 5 else
                 torch.exp(torch.clamp(p, -1.0, 1.0)) if o == 6 else
                 torch.log(torch.abs(p) + 1.0) if o == 7 else
                 torch.sqrt(p * p + 1.0) if o == 8 else torch.tanh(p))
    return torch.stack(v[-DAG_OUT:])


def _dag_grad(x, nodes, seed=0):
    x = x.detach().requires_grad_(True)
    y = _dag_value(x, nodes, seed)
    (gx,) = torch.autograd.grad(y.sum(), x)
    return y.detach(), gx


def _quad(x, u):
    Ixx, Iyy, Izz, grav = 0.01, 0.01, 0.02, 9.81
    ph, th, ps, p, q, r = x[6], x[7], x[8], x[9], x[10], x[11]
    cph, sph, cth, sth = torch.cos(ph), torch.sin(ph), torch.cos(th), torch.sin(th)
    cps, sps = torch.cos(ps), torch.sin(ps)
    w = q * sph + r * cph
    return torch.stack([
        x[3], x[4], x[5], u[0] * (cph * sth * cps + sph * sps),
        u[0] * (cph * sth * sps - sph * cps), u[0] * (cph * cth) - grav, p + w * (sth / cth),
        q * cph - r * sph, w / cth, (u[1] + (Iyy - Izz) * q * r) / Ixx,
        (u[2] + (Izz - Ixx) * p * r) / Iyy, (u[3] + (Ixx - Iyy) * p * q) / Izz])


def _kkt_exact(x, K):
    """Constraint Jacobian and Hessian of the Lagrangian, interval by interval, as (K, 12, 16,
    n) and (K, 16, 16, n) blocks."""
    w, _, lam_f, lam = x
    n = w.shape[1]
    z = w[:16 * K].reshape(K, 16, n)
    mult = lam[12:].reshape(K, 12, n)

    def step(v):
        return _rk4(_quad, v[:12], v[12:], 0.05)

    def gamma(v, m, f):
        return (step(v) * m).sum() + f * ((v[:12] ** 2).sum() + 0.1 * (v[12:] ** 2).sum())

    J, H = [], []
    jac = torch.func.vmap(torch.func.jacrev(step))
    hess = torch.func.vmap(torch.func.hessian(gamma))
    per = max(1, min(K, 40000 // n))
    for k in range(0, K, per):
        zz = z[k:k + per].permute(0, 2, 1).reshape(-1, 16)
        mm = mult[k:k + per].permute(0, 2, 1).reshape(-1, 12)
        ff = lam_f[0].repeat(zz.shape[0] // n)
        J.append(jac(zz).reshape(-1, n, 12, 16).permute(0, 2, 3, 1))
        H.append(hess(zz, mm, ff).reshape(-1, n, 16, 16).permute(0, 2, 3, 1))
    J, H = torch.cat(J), torch.cat(H)
    kkt = _kkt(K)  # the order of the nonzeros
    r, c = (torch.as_tensor(np.asarray(v).astype(np.int64)).to(DEV)
            for v in (kkt.jac_pattern.row, kkt.jac_pattern.col()))
    k, i = (r - 12).div(12, rounding_mode="floor"), (r - 12) % 12
    inside = (r >= 12) & (c.div(16, rounding_mode="floor") == k)
    jv = J[k.clamp(min=0), i, (c - 16 * k).clamp(0, 15)]
    other = torch.where(r < 12, 1.0, -1.0)[:, None].to(F64).expand(-1, n)
    jv = torch.where(inside[:, None], jv, other)
    r, c = (torch.as_tensor(np.asarray(v).astype(np.int64)).to(DEV)
            for v in (kkt.hess_pattern.row, kkt.hess_pattern.col()))
    return [jv, H[r.div(16, rounding_mode="floor"), r % 16, c % 16]]


def exact(case, seed):
    kind, x = case["kind"], _inputs(case, seed)
    if kind == "eval":
        if case["tape"] == "step":
            return [_rk4(_ode, x[0], x[1][0], 0.02)]
        return list(_rollout(x[0], x[1]))
    if kind == "dag_sparsity":
        return None
    if kind == "dag_adjoint":
        y, gx = _dag_grad(x[0], case["nodes"])
        return [y], [gx[None]]
    if kind == "batch":
        items = _mixed_items(case["total"])
        got = {}
        for nodes in sorted({k for k, _ in items}):
            at = [i for i, (k, _) in enumerate(items) if k == nodes]
            y, gx = _dag_grad(torch.cat([x[i] for i in at], 1), nodes)
            sizes = [items[i][1] for i in at]
            for i, yy, gg in zip(at, y.split(sizes, 1), gx.split(sizes, 1)):
                got[i] = ([yy], [gg[None]])
        return [got[i] for i in range(len(items))]
    if kind == "kkt":
        return _kkt_exact(x, case["intervals"])
    if kind == "mapsum":
        x0, u = x[0].requires_grad_(True), x[1].requires_grad_(True)
        xn, cost = _rollout(x0, u[:, None])
        gx, gu = torch.autograd.grad(cost.sum(), (x0, u))
        return [xn.detach(), cost.detach().sum(1)], [gx[None], gu[None]]
    x0, u = x[0].requires_grad_(True), x[1].requires_grad_(True)
    xn, cost = _rollout(x0, u)
    if kind == "autograd":
        gx, gu = torch.autograd.grad(cost.sum(), (x0, u))
        return xn.detach(), cost.detach(), gx, gu
    J = torch.stack([torch.cat(r) for r in _rows(list(xn), (x0, u))], 1)  # (4+S, 4, n)
    (gx, gu), = _rows([cost], (x0, u))
    if kind == "forward":
        sd = torch.cat(x[2:], 1)  # (nfwd, 4+S, n)
        fx = torch.stack([(J * s[:, None]).sum(0) for s in sd])
        fc = torch.stack([(torch.cat([gx, gu]) * s).sum(0, keepdim=True) for s in sd])
        return [xn.detach(), cost.detach()], [fx, fc]
    if kind == "host":
        res = [xn.detach().T.contiguous().cpu().numpy(), cost.detach().T.contiguous().cpu().numpy()]
        jac = J.permute(2, 0, 1).contiguous().cpu().numpy()
        return res, [jac, None], [gx.T[:, None].contiguous().cpu().numpy(),
                                  gu.T[:, None].contiguous().cpu().numpy()]
    return [xn.detach(), cost.detach()], [J, None], [gx[None], gu[None]]
