"""The work that a program built on this framework has it do, as cases that can be timed and compared.

Two groups.  The codec calls run a whole proxy call as a program or the chunk server makes it: the
stream's temporal context comes in, one chunk or frame is coded, the context goes out.  The layer
calls run the operators that the networks of those codecs are made of, at the pixel counts and
channel widths of those networks, through `dcvc_b200.ops`; a network's pixel count is that of the
1/8 grid (1920x1080: 136 x 240 = 32640, 3840x2160: 270 x 480 = 129600, 416x240: 30 x 52 = 1560) or
of the 1/16 grid of its entropy-parameter path.

A case is a dict: `op` names the call, the other entries are its sizes and options.
"""
import functools

import numpy as np
import torch

from dcvc_b200 import _native as N
from dcvc_b200 import ops
from dcvc_b200.entropy_tables import add_cdf_to_state_dict
from dcvc_b200.inference_extensions_cuda import DMCHTSProxy, DMCIProxy, DMCLDProxy
from dcvc_b200.model_spec import perturbed_dmci_state_dict, perturbed_hts_state_dict, perturbed_ld_state_dict
from dcvc_b200.synthetic import padding_for

SKIP_THRESHOLD = 0.15
FRAMES = 8
EPILOGUES = {"bias": N.EPI_BIAS, "wsilu": N.EPI_BIAS_WSILU, "res": N.EPI_BIAS_RES, "res_q": N.EPI_BIAS_RES_Q,
             "quad": N.EPI_QUAD}
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16}
# resolutions of the serving mix (416x240 .. 3840x2160), height x width
SIZES = ((240, 416), (480, 832), (720, 1280), (1080, 1920), (2160, 3840))


def listed():
    return [
        # one 8-frame 1080p chunk of a running stream, the headline workload, in each direction
        {"name": "hts_encode_1080p", "op": "hts_encode", "h": 1080, "w": 1920, "qp": 42, "precision": "fp16"},
        {"name": "hts_decode_1080p", "op": "hts_decode", "h": 1080, "w": 1920, "qp": 21, "precision": "fp16"},
        # one frame of a low-delay call's receiving end
        {"name": "ld_decode_720p", "op": "ld_decode", "h": 720, "w": 1280, "qp": 30},
        # the smallest whole call: a 256x256 intra frame, bound by launches and round trips
        {"name": "intra_encode_256", "op": "intra_encode", "h": 256, "w": 256, "qp": 32},
        # ConvFFN of a 512-channel block (HT-S transforms) at 1080p
        {"name": "ffn_512_1080p", "op": "ffn", "m": 32640, "c": 512, "cffn": 256},
        # ConvFFN of a 256-channel block (low-delay codec) on an odd pixel count
        {"name": "ffn_256_odd", "op": "ffn", "m": 67 * 119, "c": 256, "cffn": 128},
        # ffn.0 of a 512-channel block: the largest layer, at 2160p, and its 8-bit form at 1080p
        {"name": "quad_2160p", "op": "conv1x1", "epi": "quad", "m": 129600, "n": 1024, "k": 512, "dtype": "f16"},
        {"name": "quad_f8_1080p", "op": "conv1x1_f8", "epi": "quad", "m": 32640, "n": 1024, "k": 512},
        # dc.3 of a 512-channel block, bound by memory
        {"name": "res_1080p", "op": "conv1x1", "epi": "res", "m": 32640, "n": 512, "k": 256, "dtype": "f16"},
        # dc.0 of a 512-channel block of a packed batch: three 720p streams in the BF16 form
        {"name": "wsilu_bf16_720p", "op": "conv1x1", "epi": "wsilu", "m": 43200, "n": 256, "k": 512,
         "dtype": "bf16"},
        # a layer of the prior fusion at the smallest resolution: bound by latency
        {"name": "res_768_240p", "op": "conv1x1", "epi": "res", "m": 390, "n": 768, "k": 768, "dtype": "f16"},
        # the depthwise 3x3 of a 512-channel block at 2160p
        {"name": "dwconv_2160p", "op": "dwconv", "h": 270, "w": 480, "c": 256, "images": 1, "dtype": "f16"},
    ]


def draw(rng):
    """One more case of the ranges above."""
    op = rng.choice(["hts_encode", "hts_decode", "ld_decode", "intra_encode", "ffn", "ffn", "conv1x1", "conv1x1",
                     "conv1x1", "conv1x1_f8", "dwconv", "dwconv"])

    def log_uniform(lo, hi):
        return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))

    if op in ("hts_encode", "hts_decode", "ld_decode", "intra_encode"):
        h, w = rng.choice(SIZES[:4])
        if rng.random() < 0.5:  # cropped content: any even size below the standard one
            h, w = 2 * (rng.randint(h * 3 // 4, h) // 2), 2 * (rng.randint(w * 3 // 4, w) // 2)
        case = {"op": op, "h": h, "w": w, "qp": rng.randint(0, 63)}
        if op.startswith("hts"):
            case["precision"] = rng.choice(["fp16", "fp16", "bf16", "fp8"])
        return case
    if op == "dwconv":
        return {"op": op, "h": log_uniform(15, 270), "w": log_uniform(26, 480),
                "c": rng.choice([128, 256, 256, 384, 512]) // (2 if rng.random() < 0.2 else 1), "images": 1,
                "dtype": rng.choice(["f16", "bf16"])} if rng.random() < 0.7 else {
                    "op": op, "h": log_uniform(15, 68), "w": log_uniform(26, 240), "c": rng.choice([256, 512]),
                    "images": rng.randint(2, 4), "dtype": rng.choice(["f16", "bf16"])}
    m = log_uniform(390, 129600)
    if op == "ffn":
        c, cffn = rng.choice([(512, 256), (512, 256), (256, 256), (256, 128)])
        return {"op": op, "m": m, "c": c, "cffn": cffn}
    if op == "conv1x1_f8":
        return {"op": op, "epi": "quad", "m": m, "n": 1024, "k": rng.choice([256, 512])}
    epi = rng.choice(["bias", "wsilu", "res", "res_q", "quad"])
    if epi == "quad":
        n, k = rng.choice([(1024, 512), (1024, 256), (512, 256), (1536, 384)])
    elif epi == "wsilu":
        n, k = rng.choice([(256, 512), (256, 256), (128, 256), (384, 384)])
    elif epi == "bias":
        n, k = rng.choice([(512, 1024), (256, 512), (192, 256), (512, 2048)])
    else:
        n, k = rng.choice([(512, 256), (256, 256), (256, 128), (512, 512), (768, 768)])
    if epi == "bias" and k == 2048:
        m = min(m, 32640)
    return {"op": op, "epi": epi, "m": m, "n": n, "k": k, "dtype": rng.choice(["f16", "f16", "bf16"])}


# ------------------------------------------------------------------------------ inputs


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _video(h, w, frames, seed):
    """[1, 3 * frames, h, w] model input of synthetic 8-bit 4:2:0 video: sinusoid fields, a textured
    patch moving by (1, 2) pixels a frame, sensor noise; chroma up-sampled to the luma grid, /255 - 0.5."""
    g = _generator(seed)

    def uniform(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, device="cuda", generator=g)

    def field(hh, ww, amplitude):
        yy = torch.arange(hh, device="cuda", dtype=torch.float32)[:, None]
        xx = torch.arange(ww, device="cuda", dtype=torch.float32)[None, :]
        out = torch.zeros(hh, ww, device="cuda")
        for period, theta, phase in zip(uniform(16, 128, 4), uniform(0, 3.14159, 4), uniform(0, 6.28318, 4)):
            f = 6.28318 / period
            out += torch.sin(f * (torch.cos(theta) * xx + torch.sin(theta) * yy) + phase)
        return 128 + amplitude * out / 4

    h2, w2 = (h + 1) // 2, (w + 1) // 2
    y0, c0 = field(h, w, 60.0), torch.stack([field(h2, w2, 20.0), field(h2, w2, 20.0)])
    ps = min(256, h // 2, w // 2)
    patch = uniform(0, 255, ps, ps)
    planes = []
    for t in range(frames):
        y = y0 + 0.5 * t
        top, left = (h // 4 + t) % (h - ps), (w // 4 + 2 * t) % (w - ps)
        y[top:top + ps, left:left + ps] = patch
        y = y + 2.0 * torch.randn(h, w, device="cuda", generator=g)
        c = c0.repeat_interleave(2, 1).repeat_interleave(2, 2)[:, :h, :w]
        planes += [y[None], c]
    x = torch.cat(planes).round_().clamp_(0, 255).to(torch.float16)[None]
    x = x / 255.0 - 0.5
    return x.contiguous(memory_format=torch.channels_last)


def _reference(x):
    """The first frame of a clip on the codec's padded grid: what seeds a stream's temporal context."""
    pr, pb = padding_for(x.shape[2], x.shape[3])
    f = torch.nn.functional.pad(x[:, :3].float(), (0, pr, 0, pb), mode="replicate").half()
    return f.contiguous(memory_format=torch.channels_last)


@functools.lru_cache(maxsize=None)
def _weights(model):
    sd = {"hts": perturbed_hts_state_dict, "ld": perturbed_ld_state_dict, "intra": perturbed_dmci_state_dict}[model](0)
    sd = add_cdf_to_state_dict(sd)
    return {k: (v.half().cuda() if v.is_floating_point() else v) for k, v in sd.items()}


@functools.lru_cache(maxsize=None)
def _hts_parameters(precision):
    """The one parameter set that a program keeps for all its streams of a form."""
    p = DMCHTSProxy(precision)
    p.set_param(_weights("hts"), SKIP_THRESHOLD)
    return p


def _hts(precision):
    p = DMCHTSProxy(precision)
    p.share_params_from(_hts_parameters(precision))
    return p


def prepare(case, seed):
    op = case["op"]
    if op in ("hts_encode", "hts_decode", "ld_decode", "intra_encode"):
        return _prepare_codec(case, seed)
    g = _generator(seed)

    def rnd(*shape, scale=1.0, dtype=torch.float16):
        return (scale * torch.randn(*shape, device="cuda", generator=g)).to(dtype)

    s = {"case": dict(case)}
    if op == "dwconv":
        dtype = DTYPES[case["dtype"]]
        s["h"], s["w"], s["img_h"] = case["h"] * case["images"], case["w"], case["h"]
        s["x"] = rnd(s["h"] * s["w"], case["c"], dtype=dtype)
        s["weight"] = rnd(9, case["c"], scale=1 / 3, dtype=torch.float32)
        return s
    if op == "ffn":
        m, c, cffn = case["m"], case["c"], case["cffn"]
        s["x"] = rnd(m, c)
        s["w1"], s["b1"] = rnd(4 * cffn, c, scale=c ** -0.5), rnd(4 * cffn, scale=0.1, dtype=torch.float32)
        s["w2"], s["b2"] = rnd(c, cffn, scale=cffn ** -0.5), rnd(c, scale=0.1, dtype=torch.float32)
        return s
    m, n, k = case["m"], case["n"], case["k"]
    s["epi"] = EPILOGUES[case["epi"]]
    s["bias"] = rnd(n, scale=0.1, dtype=torch.float32)
    if op == "conv1x1_f8":
        w = rnd(n, k, scale=k ** -0.5, dtype=torch.float32)
        s["a"] = rnd(m, k, dtype=torch.float32).to(torch.float8_e4m3fn)
        s["wscale"] = (w.abs().amax(1) / 448.0).contiguous()
        s["weight"] = (w / s["wscale"][:, None]).to(torch.float8_e4m3fn)
        return s
    dtype = DTYPES[case["dtype"]]
    s["a"], s["weight"] = rnd(m, k, dtype=dtype), rnd(n, k, scale=k ** -0.5, dtype=dtype)
    s["res"] = rnd(m, n, dtype=dtype) if case["epi"].startswith("res") else None
    s["q"] = (1 + 0.25 * (2 * torch.rand(n, device="cuda", generator=g) - 1)).to(dtype) if case["epi"] == "res_q" \
        else None
    return s


def _prepare_codec(case, seed):
    h, w, qp, op = case["h"], case["w"], case["qp"], case["op"]
    pr, pb = padding_for(h, w)
    s = {"case": dict(case), "pr": pr, "pb": pb, "filled": 0}
    if op.endswith("encode"):  # room for a quarter of the chunk's raw 4:2:0 size
        s["packet"] = np.zeros((h + pb) * (w + pr) * 3 // 8 * (FRAMES if op == "hts_encode" else 1), np.uint8)
    if op == "intra_encode":
        s["x"] = _video(h, w, 1, seed)
        s["proxy"] = DMCIProxy()
        s["proxy"].set_param(_weights("intra"), SKIP_THRESHOLD)
        return s
    if op == "ld_decode":
        clip = _video(h, w, 2, seed)
        s["ref"] = _reference(clip)
        enc, s["proxy"] = DMCLDProxy(), DMCLDProxy()
        enc.set_param(_weights("ld"), SKIP_THRESHOLD)
        s["proxy"].set_param(_weights("ld"), SKIP_THRESHOLD)
        enc.add_ref_feature_from_frame(s["ref"], True)
        x = clip[:, 3:].contiguous(memory_format=torch.channels_last)
        s["bits"], s["ecp"] = enc.compress(x, qp, False, pb, pr)
        s["proxy"].add_ref_feature_from_frame(s["ref"], False)
        return s
    # a stream that has coded one chunk: the second one is what is measured
    clip = _video(h, w, 2 * FRAMES, seed)
    first, second = (clip[:, i * 3 * FRAMES:(i + 1) * 3 * FRAMES].contiguous(memory_format=torch.channels_last)
                     for i in (0, 1))
    enc = _hts(case["precision"])
    enc.add_ref_feature_from_frame(_reference(clip), True)
    bits, ecp = enc.compress(first, qp, False, pb, pr)
    if op == "hts_encode":
        s["proxy"], s["x"] = enc, second
    else:
        s["bits"], s["ecp"] = enc.compress(second, qp, False, pb, pr)
        s["proxy"] = _hts(case["precision"])
        s["proxy"].add_ref_feature_from_frame(_reference(clip), False)
        s["proxy"].decompress(bits, qp, h, w, ecp, False)
    s["context"], s["flags"] = s["proxy"].export_state()
    s["after"] = torch.empty_like(s["context"])
    return s


# ------------------------------------------------------------------------------ one pass


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "hts_encode":
        # the chunk server's encode request: context in, chunk coded, context out
        p = s["proxy"]
        p.import_state(s["context"], s["flags"])
        bits, ecp = p.compress(s["x"], case["qp"], False, s["pb"], s["pr"])
        p.export_state(s["after"])
        return {"packet": _packet(s, bits), "size": bits.size, "ec_parallel": ecp,
                "context": _as_activations(s["after"], case)}
    if op == "hts_decode":
        p = s["proxy"]
        p.import_state(s["context"], s["flags"])
        frames = p.decompress(s["bits"], case["qp"], case["h"], case["w"], s["ecp"], False)
        p.export_state(s["after"])
        return {"frames": [_keeping(f, p) for f in frames], "context": _as_activations(s["after"], case)}
    if op == "ld_decode":
        # the first predicted frame after a key frame
        s["proxy"].add_ref_feature_from_frame(s["ref"], False)
        x_hat = s["proxy"].decompress(s["bits"], case["qp"], case["h"], case["w"], s["ecp"], False)
        return _keeping(x_hat, s["proxy"])
    if op == "intra_encode":
        bits, x_hat, ecp = s["proxy"].compress(s["x"], case["qp"], s["pb"], s["pr"])
        return {"packet": _packet(s, bits), "size": bits.size, "ec_parallel": ecp,
                "x_hat": _keeping(x_hat, s["proxy"])}
    if op == "dwconv":
        if case["images"] == 1 and case["dtype"] == "f16":
            return ops.dwconv3x3(s["x"], s["h"], s["w"], s["weight"])
        return ops.dwconv3x3_ex(s["x"], s["h"], s["w"], s["weight"], img_h=s["img_h"])
    if op == "ffn":
        return ops.conv_ffn(s["x"], s["w1"], s["b1"], s["w2"], s["b2"])
    if op == "conv1x1_f8":
        return ops.conv1x1_f8(s["a"], s["weight"], s["wscale"], s["bias"], s["epi"])
    return ops.conv1x1(s["a"], s["weight"], s["bias"], s["epi"], res=s["res"], qscale=s["q"])


def _packet(s, bits):
    """The payload in the program's packet buffer, zeros behind it."""
    s["packet"][:bits.size] = bits
    s["packet"][bits.size:s["filled"]] = 0
    s["filled"] = bits.size
    return s["packet"]


def _keeping(frame, proxy):
    """The frame, a view of the proxy's own buffer, with the proxy kept alive as long as the frame is."""
    frame._proxy = proxy
    return frame


def _as_activations(state, case):
    return state.view(torch.float16 if case["precision"] == "fp16" else torch.bfloat16)


# ------------------------------------------------------------------------------ what a pass cannot do without

# multiply-accumulates per pixel of the 1/8 grid and bytes of the 16-bit weights of the call that the case
# makes: the 1x1 and 3x3 layers it runs, each at its own scale
_CODEC_MACS = {"hts_encode": 34.87e6, "hts_decode": 47.71e6, "ld_decode": 4.53e6, "intra_encode": 29.08e6}
_CODEC_WEIGHTS = {"hts_encode": 2 * 57.1e6, "hts_decode": 2 * 67.8e6, "ld_decode": 2 * 7.0e6,
                  "intra_encode": 2 * 41.9e6}


def work(case):
    op = case["op"]
    if op in _CODEC_MACS:
        pr, pb = padding_for(case["h"], case["w"])
        pixels = (case["h"] + pb) * (case["w"] + pr)
        grid = pixels // 64
        frames = FRAMES if op.startswith("hts") else 1
        context = 2 * grid * (1024 + 512 + 192) * 2 if op.startswith("hts") else 0
        return {"bytes": 2 * 3 * frames * pixels + context + _CODEC_WEIGHTS[op], "flops": 2 * _CODEC_MACS[op] * grid}
    if op == "dwconv":
        n = case["h"] * case["images"] * case["w"] * case["c"]
        return {"bytes": 4 * n + 36 * case["c"], "flops": 18 * n}
    if op == "ffn":
        m, c, f = case["m"], case["c"], case["cffn"]
        return {"bytes": 4 * m * c + 2 * 5 * c * f + 4 * (4 * f + c), "flops": 2 * m * 5 * c * f}
    m, n, k = case["m"], case["n"], case["k"]
    nout = n // 4 if case["epi"] == "quad" else n
    esz = 1 if op == "conv1x1_f8" else 2
    res = m * n if case["epi"].startswith("res") else 0
    return {"bytes": esz * (m * k + n * k) + 2 * (m * nout + res) + 4 * n * (2 if esz == 1 else 1),
            "flops": 2 * m * n * k}


# ------------------------------------------------------------------------------ the same in 64 bits


def _wsilu(x):
    return x * torch.sigmoid(4 * x)


def exact(case, seed):
    op = case["op"]
    if op in _CODEC_MACS:
        return None  # a payload and a chain of some hundred layers: no 64-bit form outside a full codec
    s = prepare(case, seed)
    if op == "dwconv":
        x = s["x"].double().reshape(case["images"], case["h"], case["w"], case["c"]).permute(0, 3, 1, 2)
        wt = s["weight"].double().t().reshape(case["c"], 3, 3)
        pad = torch.nn.functional.pad(x, (1, 1, 1, 1))
        out = torch.zeros_like(x)
        for ky in range(3):
            for kx in range(3):
                out += pad[:, :, ky:ky + case["h"], kx:kx + case["w"]] * wt[None, :, ky, kx, None, None]
        return out.permute(0, 2, 3, 1).reshape(s["h"] * s["w"], case["c"])
    if op == "ffn":
        x = s["x"].double()
        q = _wsilu(x @ s["w1"].double().t() + s["b1"].double()).reshape(x.shape[0], case["cffn"], 4).sum(2)
        return q @ s["w2"].double().t() + s["b2"].double() + x
    if op == "conv1x1_f8":
        v = (s["a"].float().double() @ s["weight"].float().double().t()) * s["wscale"].double() + s["bias"].double()
    else:
        v = s["a"].double() @ s["weight"].double().t() + s["bias"].double()
    if case["epi"] == "quad":
        return _wsilu(v).reshape(v.shape[0], case["n"] // 4, 4).sum(2)
    if case["epi"] == "wsilu":
        return _wsilu(v)
    if case["epi"] == "res":
        return v + s["res"].double()
    if case["epi"] == "res_q":
        return (v + s["res"].double()) * s["q"].double()
    return v
