"""The forms of the GEMM that the library takes by itself.  Bias and WSiLU on CTA pairs (block_n = 0): bitwise the one-CTA tiles
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


@pytest.mark.parametrize("M,Nn,K", [(1, 64, 64), (127, 256, 64), (129, 512, 128), (256, 512, 192), (300, 768, 256), (257, 1024, 320),
                                    (390, 768, 384), (1024, 512, 448), (1000, 384, 512), (2304, 256, 576), (2305, 256, 1536)])
@pytest.mark.parametrize("epi", [N.EPI_BIAS, N.EPI_BIAS_WSILU, N.EPI_BIAS_RES, N.EPI_BIAS_RES_Q, N.EPI_BIAS_RES2, N.EPI_QUAD, N.EPI_BIAS_Q,
                                 N.EPI_SUBPEL])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_narrow_tiles(M, Nn, K, epi, dtype):
    """GEMMs small enough for the 32-column tiles (and, last, one row tile too many), with every split of the
    K blocks into stages: bitwise the widest tile that N allows."""
    g = torch.Generator(device="cuda").manual_seed(M + Nn + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(Nn, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    b = torch.randn(Nn, device="cuda", generator=g) * 0.3
    res, res2 = (torch.randn(M, Nn, device="cuda", generator=g).to(dtype) for _ in range(2))
    q = (torch.rand(Nn, device="cuda", generator=g) + 0.5).to(dtype)
    args = dict(res=res, res2=res2, qscale=q)
    wide = next(bn for bn in (256, 128, 64) if Nn % bn == 0)
    if epi == N.EPI_SUBPEL:
        args = dict(sub_w=M, sub_cout=Nn)
        w = torch.cat([w, -w, 2 * w, w.flip(0)])
    elif epi == N.EPI_QUAD and wide != 256:
        pytest.skip("the quad GEMM has 256 columns or a multiple")
    ref = ops.conv1x1(a, w, b, epi, block_n=wide, **args)
    out = ops.conv1x1(a, w, b, epi, **args)
    torch.cuda.synchronize()
    assert N.device_error() == 0
    assert torch.equal(out.view(torch.int16), ref.view(torch.int16))


def test_narrow_tiles_are_the_librarys_choice():
    a = torch.zeros(128, 64, device="cuda", dtype=torch.float16)
    w = torch.zeros(256, 64, device="cuda", dtype=torch.float16)
    b = torch.zeros(256, device="cuda")
    with pytest.raises(N.DcvcError):
        ops.conv1x1(a, w, b, block_n=32)
    with pytest.raises(N.DcvcError):
        ops.conv1x1(a, w[:96].contiguous(), b)  # no width for N = 96


@pytest.mark.parametrize("M,Nn,K", [(4737, 512, 512), (8160, 512, 512), (8193, 512, 576), (9473, 512, 512), (8160, 768, 768), (19000, 256, 512), (19073, 256, 1024),
                                    (6240, 768, 768), (9601, 512, 448)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("with_q", [False, True])
def test_residual_pairs(M, Nn, K, dtype, with_q):
    """The residual epilogues on CTA pairs, and around the sizes where the library takes them."""
    g = torch.Generator(device="cuda").manual_seed(M + Nn + K)
    a = torch.randn(M, K, device="cuda", generator=g).to(dtype)
    w = (torch.randn(Nn, K, device="cuda", generator=g) * K ** -0.5).to(dtype)
    b = torch.randn(Nn, device="cuda", generator=g) * 0.3
    res = torch.randn(M, Nn + 8, device="cuda", generator=g).to(dtype)[:, 8:]
    q = (torch.rand(Nn, device="cuda", generator=g) + 0.5).to(dtype) if with_q else None
    epi = N.EPI_BIAS_RES_Q if with_q else N.EPI_BIAS_RES
    ref = ops.conv1x1(a, w, b, epi, res=res, qscale=q, block_n=128)
    buf = torch.full((M, Nn + 16), float("nan"), device="cuda", dtype=dtype)
    out = ops.conv1x1(a, w, b, epi, res=res, qscale=q, out=buf[:, 8:8 + Nn])
    torch.cuda.synchronize()
    assert N.device_error() == 0
    assert torch.equal(out.contiguous().view(torch.int16), ref.view(torch.int16))
    assert bool(torch.isnan(buf[:, :8]).all()) and bool(torch.isnan(buf[:, 8 + Nn:]).all())
    with pytest.raises(N.DcvcError):  # callers cannot ask for it
        ops.conv1x1(a, w, b, epi, res=res, qscale=q, block_n=N.BLOCK_N_PAIR)


@pytest.mark.parametrize("M", [1, 127, 390, 1000, 4736, 4737])
@pytest.mark.parametrize("C,cffn", [(512, 256), (256, 256), (256, 128)])
@pytest.mark.parametrize("with_q,in_place", [(False, False), (True, False), (False, True)])
def test_conv_ffn_of_few_pixels(M, C, cffn, with_q, in_place):
    """ConvFFN as two GEMMs, up to one row tile past its range: bitwise the tail kernel, also in place, and with
    biases that the GEMMs could not read (the one kernel takes those)."""
    g = torch.Generator(device="cuda").manual_seed(M + C + cffn)
    x = torch.randn(M, C, device="cuda", generator=g).half()
    w1 = (torch.randn(4 * cffn, C, device="cuda", generator=g) * C ** -0.5).half()
    w2 = (torch.randn(C, cffn, device="cuda", generator=g) * cffn ** -0.5).half()
    b1, b2 = (torch.randn(n + 1, device="cuda", generator=g)[1:] * 0.1 for n in (4 * cffn, C))
    q = (torch.rand(C, device="cuda", generator=g) + 0.5).half() if with_q else None
    ref = ops.dcb_tail(None, x, None, None, w1, b1, w2, b2, qscale=q)
    odd = torch.empty(C + 1, device="cuda")[1:].copy_(b2)
    assert odd.data_ptr() % 16 != 0
    aside = ops.conv_ffn(x, w1, b1, w2, odd, qscale=q)
    out = ops.conv_ffn(x, w1, b1, w2, b2, qscale=q, out=x if in_place else None)
    torch.cuda.synchronize()
    assert N.device_error() == 0
    assert torch.equal(out.view(torch.int16), ref.view(torch.int16))
    assert torch.equal(aside.view(torch.int16), ref.view(torch.int16))
