"""dcvc_gemm_pair_form(0): the library's own choice takes no kernel that works in CTA pairs - neither the pair form of
the GEMM, nor the resident quad, nor the DepthConvBlock tail - in the operators and in a codec, with the same bits as
the default, which takes them.  Which kernels ran is read from the profiler's kernel names."""
import re

import numpy as np
import pytest
import torch

from dcvc_b200 import _native as N
from dcvc_b200 import ops, synthetic
from tests.hts_fixtures import chunk, make_proxy, ref_frame, state_dict

pytestmark = pytest.mark.gpu

# a pair GEMM is the tiled kernel with its last template argument (PAIR) set
PAIR_KERNEL = re.compile(r"dcb_tail_kernel|quad_kernel|gemm_sm100_kernel<[^>]*true>")


@pytest.fixture(autouse=True)
def _default_form():
    yield
    N.lib.dcvc_gemm_pair_form(-1)


def _pair_kernels(call):
    """(result, names of the pair kernels that ran)"""
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        out = call()
        torch.cuda.synchronize()
    names = {e.name for e in prof.events() if "kernel" in e.name}
    assert names, "the profiler saw no kernel"
    return out, sorted(n for n in names if PAIR_KERNEL.search(n))


def _operators():
    g = torch.Generator(device="cuda").manual_seed(3)

    def rnd(*s, scale=1.0, dt=torch.float16):
        return (torch.randn(*s, device="cuda", generator=g) * scale).to(dt)

    a, b = rnd(32640, 512), rnd(1024, dt=torch.float32)
    wq, wp, res = rnd(1024, 512, scale=0.04), rnd(512, 512, scale=0.04), rnd(32640, 512)
    w2, b2 = rnd(512, 256, scale=0.06), rnd(512, dt=torch.float32)
    a8, w8 = a.float().to(torch.float8_e4m3fn), (wq.float() * 8).to(torch.float8_e4m3fn)
    ws = torch.full((1024,), 0.125, device="cuda")
    return {"quad": lambda: ops.conv1x1(a, wq, b, N.EPI_QUAD), "quad f8": lambda: ops.conv1x1_f8(a8, w8, ws, b, N.EPI_QUAD),
            "wsilu": lambda: ops.conv1x1(a, wp, b2, N.EPI_BIAS_WSILU), "bias": lambda: ops.conv1x1(a, wp, b2, N.EPI_BIAS),
            "res": lambda: ops.conv1x1(a, wp, b2, N.EPI_BIAS_RES, res=res), "conv_ffn": lambda: ops.conv_ffn(a, wq, b, w2, b2)}


@pytest.mark.parametrize("name", ["quad", "quad f8", "wsilu", "bias", "res", "conv_ffn"])
def test_operators(name):
    call = _operators()[name]
    want, pairs = _pair_kernels(call)
    assert pairs, name
    N.lib.dcvc_gemm_pair_form(0)
    got, pairs = _pair_kernels(call)
    assert pairs == [], name
    assert torch.equal(got.view(torch.int16), want.view(torch.int16))


def test_codec():
    H, W = 480, 832
    pr, pb = synthetic.padding_for(H, W)
    ref, x = ref_frame(H, W), chunk(H, W, 0)

    def run():
        enc = make_proxy(state_dict())
        enc.add_ref_feature_from_frame(ref, True)
        return enc.compress(x, 30, False, pb, pr)

    (bits, ecp), pairs = _pair_kernels(run)
    assert any("dcb_tail_kernel" in n for n in pairs)
    N.lib.dcvc_gemm_pair_form(0)
    (bits0, ecp0), pairs = _pair_kernels(run)
    assert pairs == []
    assert ecp == ecp0 and np.array_equal(bits, bits0)
