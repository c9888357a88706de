"""The native entry points of the hot operators (csrc/python/torch_calls.cpp): argument errors as the Python
wrappers raise them, the library's status as DcvcError, the caller's output and stream."""
import pytest
import torch

from dcvc_b200 import _native as N
from dcvc_b200 import ops


@pytest.mark.parametrize("call,error", [
    (lambda a, w: ops.conv1x1(a.t(), w), AssertionError),
    (lambda a, w: ops.conv1x1(a, w.t()), AssertionError),
    (lambda a, w: ops.conv1x1(a.float(), w), KeyError),
    (lambda a, w: ops.conv1x1(a, None), TypeError),
    (lambda a, w: ops.conv1x1(a, w, epilogue="bias"), TypeError),
    (lambda a, w: ops.conv1x1_f8(a[0], w, None, None), AssertionError),
    (lambda a, w: ops.conv_ffn(a, w.t(), None, w, None), AssertionError),
    (lambda a, w: ops.dwconv3x3_ex(a[0], 1, 1, w), IndexError),
    (lambda a, w: ops.dwconv3x3_ex(a.double(), 1, 1, w), KeyError),
])
def test_argument_errors(call, error):
    with pytest.raises(error):
        call(torch.zeros(4, 64, dtype=torch.float16), torch.zeros(128, 64, dtype=torch.float16))


@pytest.mark.gpu
def test_output_stream_and_status():
    a = torch.randn(300, 128, device="cuda").half()
    w = torch.randn(256, 128, device="cuda").half()
    b = torch.randn(256, device="cuda")
    ref = ops.conv1x1(a, w, b)
    assert ref.shape == (300, 256) and ref.dtype == a.dtype and not ref.requires_grad
    buf = torch.empty(300, 320, device="cuda", dtype=torch.float16)
    out = buf[:, 32:288]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            assert ops.conv1x1(a, w, b, out=out) is out  # on the capturing stream: recorded, not run
        out.fill_(float("nan"))
        graph.replay()
    side.synchronize()
    assert torch.equal(out, ref)
    with pytest.raises(N.DcvcError):
        ops.conv1x1(a[:, :100], w[:, :100].contiguous(), b)
    with pytest.raises(N.DcvcError):
        ops.conv_ffn(a, w, b, w, b)
    assert N.device_error() == 0
