"""The DepthConvBlock tail kernel (dcvc_dcb_tail): bit-identical with the separate GEMM launches it
stands for (every one of them checked against FP32 in test_gemm_gpu.py) at the edges of its tiles
(256-row pair tiles, one CTA of a pair without rows, more tiles than pairs, two rounds of tiles),
in each channel form, both types, with output pitches, in place and with per-image factors."""
import pytest
import torch

from dcvc_b200 import _native as N
from dcvc_b200 import ops

pytestmark = pytest.mark.gpu


def _inputs(M, C, cdc, cffn, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def rnd(*s, scale=1.0, dt=dtype):
        return (torch.randn(*s, device="cuda", generator=g) * scale).to(dt)

    w = [rnd(C, cdc, scale=cdc ** -0.5), rnd(C, scale=0.1, dt=torch.float32)] if cdc else [None, None]
    w += [rnd(4 * cffn, C, scale=C ** -0.5), rnd(4 * cffn, scale=0.1, dt=torch.float32),
          rnd(C, cffn, scale=cffn ** -0.5), rnd(C, scale=0.1, dt=torch.float32)]
    return rnd(M, cdc) if cdc else None, rnd(M, C), w, g


def _separate(a, x, w, q=None):
    w0, b0, w1, b1, w2, b2 = w
    y = ops.conv1x1(a, w0, b0, N.EPI_BIAS_RES, res=x) if a is not None else x
    t = ops.conv1x1(y, w1, b1, N.EPI_QUAD)
    return ops.conv1x1(t, w2, b2, N.EPI_BIAS_RES if q is None else N.EPI_BIAS_RES_Q, res=y, qscale=q)


def _same(a, b):
    torch.cuda.synchronize()
    assert N.device_error() == 0
    assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("C,cdc,cffn", [(512, 256, 256), (512, 0, 256), (256, 256, 256), (256, 0, 256),
                                        (256, 128, 128), (256, 0, 128)])
@pytest.mark.parametrize("M", [1, 100, 128, 129, 256, 257, 1000, 19200, 37889])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_equals_the_separate_launches(M, C, cdc, cffn, dtype):
    a, x, w, _ = _inputs(M, C, cdc, cffn, dtype, M + C + cdc + cffn)
    _same(ops.dcb_tail(a, x, *w), _separate(a, x, w))


@pytest.mark.parametrize("C,cdc,cffn", [(512, 256, 256), (256, 256, 256), (256, 0, 128)])
def test_in_place_with_pitch_and_factors(C, cdc, cffn):
    M, images = 3 * 700, 3
    a, x, w, g = _inputs(M, C, cdc, cffn, torch.float16, 5)
    q = (torch.rand(images, C, device="cuda", generator=g) + 0.5).half()
    ref = torch.cat([_separate(None if a is None else a[k * 700:(k + 1) * 700], x[k * 700:(k + 1) * 700], w, q[k])
                     for k in range(images)])
    buf = torch.full((M, C + 128), float("nan"), device="cuda", dtype=torch.float16)
    view = buf[:, 64:64 + C]
    view.copy_(x)
    ops.dcb_tail(a, view, *w, qscale=q, q_rows=700, out=view)
    _same(view.contiguous(), ref)
    assert torch.isnan(buf[:, :64]).all() and torch.isnan(buf[:, 64 + C:]).all()


def test_unsupported_shapes_are_refused():
    a, x, w, _ = _inputs(64, 384, 128, 128, torch.float16, 1)
    with pytest.raises(N.DcvcError):
        ops.dcb_tail(a, x, *w)
