"""The bounded waits of the DepthConvBlock tail and of the resident quad GEMM run out.  Under the stall injection the
tail's MMA warp issues nothing (its operands land, its other warps wait for MMAs that never come) and the quad loads
nothing; both CTAs of every pair wind down, the launch reports DCVC_DEVICE_TIMEOUT, and the next launch is right."""
import ctypes

import pytest
import torch

from dcvc_b200 import _native as N
from dcvc_b200 import ops

pytestmark = pytest.mark.gpu

TIMEOUT = 3  # DCVC_DEVICE_TIMEOUT


def _hooks():
    N.lib.dcvc_gemm_inject_stall.argtypes = [ctypes.c_int, ctypes.c_longlong]
    N.lib.dcvc_check_device_errors.argtypes = [ctypes.c_void_p]
    stream = torch.cuda.current_stream().cuda_stream
    return (lambda: N.lib.dcvc_gemm_inject_stall(1, 20000)), (lambda: N.lib.dcvc_check_device_errors(stream))


@pytest.mark.parametrize("C,cdc,cffn", [(512, 256, 256), (256, 256, 256), (256, 128, 128), (512, 0, 256), (256, 0, 128)])
@pytest.mark.parametrize("M", [100, 700, 19500])  # an idle odd CTA, three pairs, two tiles for some pairs
def test_tail_waits_run_out(M, C, cdc, cffn):
    g = torch.Generator(device="cuda").manual_seed(M + C + cdc)

    def rnd(*s, scale=1.0, dt=torch.float16):
        return (torch.randn(*s, device="cuda", generator=g) * scale).to(dt)

    a, x = rnd(M, cdc) if cdc else None, rnd(M, C)
    w = [rnd(C, cdc, scale=cdc ** -0.5), rnd(C, dt=torch.float32)] if cdc else [None, None]
    w += [rnd(4 * cffn, C, scale=C ** -0.5), rnd(4 * cffn, dt=torch.float32), rnd(C, cffn, scale=cffn ** -0.5),
          rnd(C, dt=torch.float32)]
    inject, check = _hooks()
    want = ops.dcb_tail(a, x, *w)
    assert check() == 0
    assert inject() == 0
    ops.dcb_tail(a, x, *w)
    assert check() == TIMEOUT
    got = ops.dcb_tail(a, x, *w)
    assert check() == 0
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


def test_conv_ffn_reports_the_tail_timeout():
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(32640, 512, device="cuda", generator=g).half()
    w1, w2 = (torch.randn(1024, 512, device="cuda", generator=g) * 0.04).half(), \
        (torch.randn(512, 256, device="cuda", generator=g) * 0.06).half()
    b1, b2 = torch.zeros(1024, device="cuda"), torch.zeros(512, device="cuda")
    inject, check = _hooks()
    want = ops.conv_ffn(x, w1, b1, w2, b2)
    assert check() == 0 and inject() == 0
    ops.conv_ffn(x, w1, b1, w2, b2)
    assert check() == TIMEOUT
    assert torch.equal(ops.conv_ffn(x, w1, b1, w2, b2), want) and check() == 0


@pytest.mark.parametrize("form,M", [("f16", 32640), ("f16", 40000), ("f8", 390), ("f8", 32640)])
def test_resident_quad_waits_run_out(form, M):
    g = torch.Generator(device="cuda").manual_seed(M)
    a, w = torch.randn(M, 512, device="cuda", generator=g), torch.randn(1024, 512, device="cuda", generator=g) * 0.04
    b = torch.randn(1024, device="cuda", generator=g) * 0.1
    if form == "f8":
        a, w, s = a.to(torch.float8_e4m3fn), w.to(torch.float8_e4m3fn), torch.ones(1024, device="cuda")

        def call(bn=0):
            return ops.conv1x1_f8(a, w, s, b, N.EPI_QUAD, block_n=bn)
    else:
        a, w = a.half(), w.half()

        def call(bn=0):
            return ops.conv1x1(a, w, b, N.EPI_QUAD, block_n=bn)
    inject, check = _hooks()
    want = call(256)
    assert check() == 0 and inject() == 0
    call()
    assert check() == TIMEOUT
    got = call()
    assert check() == 0
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))
