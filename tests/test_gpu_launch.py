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
