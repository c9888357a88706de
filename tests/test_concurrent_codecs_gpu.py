"""Several codecs at once on one GPU, at sizes where the CTA-pair kernels (DepthConvBlock tail, resident quad
GEMM, pair GEMM) run: single streams and packed batches in the three precision forms, each on its own host
thread and CUDA stream, give the bytes and frames that they give alone.  Three chunks each: the first runs
eagerly, the second records the phase graphs, the third replays them.

The work runs in a child process with a deadline, so that a launch that never ends fails the test instead of
holding the session."""
import faulthandler
import os
import subprocess
import sys
import threading

import numpy as np
import pytest
import torch

from dcvc_b200 import synthetic
from tests.hts_fixtures import SKIP_THRES, state_dict

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# (precision, height, width, packed streams)
GROUPS = [("fp8", 720, 1280, 1), ("fp16", 480, 832, 1), ("bf16", 480, 832, 4), ("bf16", 720, 1280, 3)]
CHUNKS = 3
DEADLINE = 150  # seconds; the work takes about 20


def _inputs(H, W, n):
    clips = [synthetic.video_chunk_yuv420(2 + k, H, W, 8, 0) for k in range(min(n, 2))]
    refs = [synthetic.padded_reference_frame(clips[k % len(clips)][0]) for k in range(n)]
    xs = [[synthetic.to_model_input(clips[(k + c) % len(clips)]) for k in range(n)] for c in range(CHUNKS)]
    return refs, xs


def _code(params, spec, inputs, out):
    """Codes and decodes the chunks of one group with codecs of its own; payloads and frames to `out`."""
    from dcvc_b200.inference_extensions_cuda import DMCHTSProxy
    precision, H, W, n = spec
    refs, xs = inputs
    pr, pb = synthetic.padding_for(H, W)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        enc, dec = DMCHTSProxy(precision), DMCHTSProxy(precision)
        enc.share_params_from(params[precision])
        dec.share_params_from(params[precision])
        enc.add_ref_features_from_frames(refs, True)
        dec.add_ref_features_from_frames(refs, False)
        for c in range(CHUNKS):
            qps = [(7 + 19 * k + 23 * c) % 64 for k in range(n)]
            coded = enc.compress_batch(xs[c], qps, False, pb, pr)
            frames = dec.decompress_batch([b for b, _ in coded], qps, H, W, [e for _, e in coded], False)
            out.append(([(b.tobytes(), e) for b, e in coded], [f.clone() for f in frames]))
        stream.synchronize()


def _child():
    faulthandler.dump_traceback_later(DEADLINE - 20, exit=True)
    from dcvc_b200 import _native as N
    from dcvc_b200.inference_extensions_cuda import DMCHTSProxy
    sd = state_dict()
    params = {}
    for precision in {g[0] for g in GROUPS}:
        params[precision] = DMCHTSProxy(precision)
        params[precision].set_param(sd, SKIP_THRES)
    inputs = [_inputs(*g[1:]) for g in GROUPS]
    torch.cuda.synchronize()
    print("inputs ready", flush=True)
    alone = [[] for _ in GROUPS]
    for spec, i, o in zip(GROUPS, inputs, alone):
        _code(params, spec, i, o)
    print("alone done", flush=True)
    for _ in range(2):
        together = [[] for _ in GROUPS]
        threads = [threading.Thread(target=_code, args=(params, *a)) for a in zip(GROUPS, inputs, together)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert N.device_error() == 0
        for spec, a, b in zip(GROUPS, alone, together):
            assert len(a) == len(b) == CHUNKS, spec
            for (payloads_a, frames_a), (payloads_b, frames_b) in zip(a, b):
                assert payloads_a == payloads_b, spec
                for fa, fb in zip(frames_a, frames_b):
                    assert np.array_equal(fa.view(torch.int16).cpu().numpy(), fb.view(torch.int16).cpu().numpy()), spec
        print("together done", flush=True)


def test_codecs_at_once_give_what_they_give_alone():
    r = subprocess.run([sys.executable, "-c", "from tests.test_concurrent_codecs_gpu import _child; _child()"],
                       cwd=ROOT, capture_output=True, text=True, timeout=DEADLINE)
    assert r.returncode == 0, (r.stdout + r.stderr)[-4000:]
    assert r.stdout.count("together done") == 2
