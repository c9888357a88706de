"""The bias and WSiLU GEMMs where the library takes CTA pairs by itself (block_n = 0): bitwise the one-CTA tiles
(checked against FP32 in test_gemm_gpu.py) around the point where narrower tiles stop running all at once, with a
pair whose odd CTA has no rows, a ragged last tile, the K from which pairs are taken and one below it, and a
strided output."""
import pytest
import torch

from dcvc_b200 import _native as N
from dcvc_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,Nn,K", [(18944, 256, 512), (18945, 256, 512), (19073, 256, 512), (37889, 256, 512), (9600, 512, 448),
                                    (9601, 512, 576), (8160, 768, 768), (14400, 512, 1024), (3000, 2048, 512)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("epi", [N.EPI_BIAS, N.EPI_BIAS_WSILU])
def test_same_bits(M, Nn, K, dtype, epi):
    g = torch.Generator(device="cuda").manual_seed(M + Nn + K)
    a = torch.randn(M, K + 8, device="cuda", generator=g).to(dtype)[:, 8:]
    w = (torch.randn(Nn, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    b = torch.randn(Nn, device="cuda", generator=g) * 0.3
    ref = ops.conv1x1(a, w, b, epi, block_n=256)
    buf = torch.full((M, Nn + 16), float("nan"), device="cuda", dtype=dtype)
    out = ops.conv1x1(a, w, b, epi, out=buf[:, 8:8 + Nn])
    torch.cuda.synchronize()
    assert N.device_error() == 0
    assert torch.equal(out.contiguous().view(torch.int16), ref.view(torch.int16))
    assert bool(torch.isnan(buf[:, :8]).all()) and bool(torch.isnan(buf[:, 8 + Nn:]).all())
