"""Depthwise 3x3 at the edges of its strips (8 columns x 4 rows x 64 channels): sizes around their
multiples, images of one row or column, partial channel groups, stacked images, compile-time and
run-time pitches, both types, against FP64.  Bound: the FP32 sum of nine products (each partial sum
rounded, 9 * 2^-24 of the sum of magnitudes) rounded once to the type (2^-11 or 2^-8, half a unit in
the last place, plus the smallest subnormal)."""
import pytest
import torch

from dcvc_b200 import _native as N
from dcvc_b200 import ops

pytestmark = pytest.mark.gpu


def _reference(x, wt, images, h, w):
    c = x.shape[1]
    v = x.double().reshape(images, h, w, c).permute(0, 3, 1, 2)
    k = wt.double().t().reshape(c, 1, 3, 3)
    out = torch.nn.functional.conv2d(v, k, padding=1, groups=c)
    mag = torch.nn.functional.conv2d(v.abs(), k.abs(), padding=1, groups=c)
    return [t.permute(0, 2, 3, 1).reshape(images * h * w, c) for t in (out, mag)]


@pytest.mark.parametrize("h,w,images", [(1, 1, 1), (1, 9, 2), (4, 8, 1), (5, 7, 3), (6, 17, 1), (13, 1, 2),
                                        (12, 24, 2), (33, 41, 1)])
@pytest.mark.parametrize("c,pad", [(8, 0), (64, 0), (72, 8), (128, 0), (256, 0), (256, 64), (384, 0), (512, 0), (768, 0)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_strip_edges(h, w, images, c, pad, dtype):
    g = torch.Generator(device="cuda").manual_seed(h * 1000 + w * 10 + c)
    m = images * h * w
    x = torch.randn(m, c + pad, device="cuda", generator=g).to(dtype)[:, :c]
    wt = torch.randn(9, c, device="cuda", generator=g)
    buf = torch.full((m, c + pad), float("nan"), device="cuda", dtype=dtype)
    out = ops.dwconv3x3_ex(x, images * h, w, wt, img_h=h, out=buf[:, :c])
    torch.cuda.synchronize()
    assert N.device_error() == 0
    ref, mag = _reference(x, wt, images, h, w)
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    bound = (1 + ulp) * 9 * 2.0 ** -24 * mag + ulp * ref.abs() + 2.0 ** -24
    assert bool(((out.double() - ref).abs() <= bound).all())
    assert bool(torch.isnan(buf[:, c:]).all())


@pytest.mark.parametrize("h,w,images,c", [(21, 29, 1, 256), (45, 43, 1, 512), (23, 41, 2, 512), (64, 120, 1, 128), (62, 73, 1, 384),
                                          (101, 131, 1, 768), (67, 119, 2, 256), (98, 120, 1, 264)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_strip_forms(h, w, images, c, dtype):
    """Sizes on both sides of the points where strips of two rows go from blocks of four warps to eight
    and then give way to strips of four rows."""
    test_strip_edges(h, w, images, c, 0, dtype)
