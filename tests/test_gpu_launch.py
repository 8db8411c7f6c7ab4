"""Calls without a stream argument run on torch's current stream of the current device."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [False, True])
def test_default_stream_is_torchs_current_stream(gpu_lib, side):
    import torch
    from casadi_gb300 import runtime as R, sx as S
    x = S.sym("x", 1)
    ct = R.CudaTape(S.Function("f", [x], [[x[0] * x[0] + 1.0]]))
    stream = torch.cuda.Stream() if side else torch.cuda.default_stream()
    with torch.cuda.stream(stream):
        assert (R._stream_handle(None).value or 0) == torch.cuda.current_stream().cuda_stream
        v = torch.zeros((1, 4096), dtype=torch.float64, device="cuda")
        for k in range(20):  # each call reads what the one before wrote, in stream order
            v, = ct.eval([v * 0.0 + k])
        got = v.cpu()
    assert (got == 19.0 * 19.0 + 1.0).all()
    ct.sync()


@pytest.mark.parametrize("residence", [0, 2, 3])
@pytest.mark.parametrize("call", ["eval", "reverse", "sp_forward"])
def test_two_threads_evaluate_one_tape(gpu_lib, call, residence):
    """Launches of the same kernels with different shared memory sizes (CTA shapes and team sizes
    follow the launch size) from two host threads on two streams: no call fails, and the results have
    the bits of the same calls made alone."""
    import ctypes as ct
    import threading

    import torch
    from casadi_gb300 import runtime as R, workloads as W
    lib = R.load()
    f = W.cartpole_rollout(2)
    t = R.CudaTape(f)
    t.set_residence(residence)
    bits = dict(dtype=torch.int64, device="cuda")
    jobs = []
    for n in (131072, 1001):
        if call == "sp_forward":
            args = [torch.randint(0, 1 << 62, (k, n), **bits) for k in f.tape.nnz_in]
        else:
            args = [torch.from_numpy(a).cuda() for a in W.cartpole_inputs(n, steps=2, seed=n)]
        seeds = [torch.ones((1, k, n), dtype=torch.float64, device="cuda") for k in f.tape.nnz_out]
        out = t._outs(t.nnz_out, n), t._outs(t.nnz_in, n, 1)
        scratch = torch.empty(max(t.scratch_bytes(n), 8), dtype=torch.uint8, device="cuda")
        jobs.append((n, args, seeds, out, scratch))

    def run(job, stream, times):
        n, args, seeds, (res, asens), scratch = job
        a, r, s, x = (R._ptr_array(v) for v in (args, res, seeds, asens))
        h = R._stream_handle(stream)
        for _ in range(times):
            if call == "eval":
                st = lib.casadi_gb300_eval(t.id, n, n, a, r, h)
            elif call == "sp_forward":
                st = lib.casadi_gb300_sp_forward(t.id, n, n, a, r, h)
            else:
                st = lib.casadi_gb300_reverse(t.id, n, n, 1, a, r, s, x,
                                              ct.c_void_p(scratch.data_ptr()), scratch.numel(), h)
            R.check(st)
        return [v.view(torch.int64) for v in (res + asens if call == "reverse" else res)]

    want = [[v.clone() for v in run(j, torch.cuda.current_stream(), 2)] for j in jobs]
    torch.cuda.synchronize()
    errors = []

    def work(job, ref):
        try:
            s = torch.cuda.Stream()
            for _ in range(10):
                got = run(job, s, 200)
                s.synchronize()
                for g, w in zip(got, ref):
                    if not bool((g == w).all()):
                        raise AssertionError("n = %d: other bits" % job[0])
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=a) for a in zip(jobs, want)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not errors, errors
    t.sync()
