"""The quad GEMM with resident activations at sizes from which the library takes it (six units of 256 rows x 256
columns per pair of SMs): bitwise the tiled kernel around that point, with a ragged last row tile, ranges that start
inside a row tile, one and two row tiles of slabs, K from one block to eight, and pitches that allow and forbid
32-byte stores."""
import pytest
import torch

from dcvc_b200 import _native as N
from dcvc_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,Nn,K", [(28160, 1024, 512), (28161, 1024, 512), (28417, 1024, 448), (18689, 1536, 384),
                                    (14209, 2048, 512), (43000, 768, 256), (57000, 512, 128), (113500, 256, 64)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_same_bits_as_the_tiled_kernel(M, Nn, K, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + Nn + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(Nn, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    b = torch.randn(Nn, device="cuda", generator=g) * 0.3
    ref = ops.conv1x1(a, w, b, N.EPI_QUAD, block_n=256)
    out = ops.conv1x1(a, w, b, N.EPI_QUAD)
    buf = torch.full((M, Nn // 4 + 24), float("nan"), device="cuda", dtype=dtype)
    odd = ops.conv1x1(a, w, b, N.EPI_QUAD, out=buf[:, 8:8 + Nn // 4])
    torch.cuda.synchronize()
    assert N.device_error() == 0
    assert torch.equal(out.view(torch.int16), ref.view(torch.int16))
    assert torch.equal(odd.contiguous().view(torch.int16), ref.view(torch.int16))
    assert bool(torch.isnan(buf[:, :8]).all()) and bool(torch.isnan(buf[:, 8 + Nn // 4:]).all())
