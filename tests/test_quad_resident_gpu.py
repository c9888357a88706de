"""The quad GEMM's form with resident activations (the library's choice, block_n = 0): bitwise the tiled
kernel (checked against FP32 in test_gemm_gpu.py) at the edges of its tiles (256-row pair tiles, one
CTA of the pair without rows), of its work split (fewer units than pairs, ranges that start inside a row
tile), with one and two row tiles of slabs in shared memory, in each type, and with output pitches that
allow and forbid 32-byte stores."""
import pytest
import torch

from dcvc_b200 import _native as N
from dcvc_b200 import ops

pytestmark = pytest.mark.gpu


def _same(a, b):
    torch.cuda.synchronize()
    assert N.device_error() == 0
    assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("M,Nn,K", [(1, 256, 64), (128, 1024, 512), (129, 1024, 512), (257, 512, 448), (6400, 1024, 512),
                                    (9500, 2048, 512), (9601, 1024, 512), (12700, 1024, 448), (19000, 1536, 384), (25000, 1024, 256), (33000, 256, 128)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_16_bit(M, Nn, K, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + Nn + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(Nn, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    b = torch.randn(Nn, device="cuda", generator=g) * 0.3
    ref = ops.conv1x1(a, w, b, N.EPI_QUAD, block_n=256)
    _same(ops.conv1x1(a, w, b, N.EPI_QUAD), ref)
    buf = torch.full((M, Nn // 4 + 24), float("nan"), device="cuda", dtype=dtype)
    out = ops.conv1x1(a, w, b, N.EPI_QUAD, out=buf[:, 8:8 + Nn // 4])
    _same(out.contiguous(), ref)
    assert bool(torch.isnan(buf[:, :8]).all()) and bool(torch.isnan(buf[:, 8 + Nn // 4:]).all())


@pytest.mark.parametrize("M,Nn,K", [(1, 256, 256), (200, 1024, 512), (9600, 1024, 512), (19100, 512, 768), (33000, 1024, 256)])
def test_e4m3(M, Nn, K):
    g = torch.Generator(device="cuda").manual_seed(M + Nn + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(torch.float8_e4m3fn)
    w = torch.randn(Nn, K, device="cuda", generator=g) * K ** -0.5
    ws = (w.abs().amax(1) / 448.0).contiguous()
    wq = (w / ws[:, None]).to(torch.float8_e4m3fn)
    b = torch.randn(Nn, device="cuda", generator=g) * 0.3
    _same(ops.conv1x1_f8(a, wq, ws, b, N.EPI_QUAD), ops.conv1x1_f8(a, wq, ws, b, N.EPI_QUAD, block_n=256))


def test_form_is_not_selectable_by_callers():
    a = torch.zeros(128, 64, device="cuda", dtype=torch.float16)
    w = torch.zeros(256, 64, device="cuda", dtype=torch.float16)
    with pytest.raises(N.DcvcError):
        ops.conv1x1(a, w, torch.zeros(256, device="cuda"), N.EPI_QUAD, block_n=-3)
