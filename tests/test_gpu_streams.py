"""A runner's buffers are zeroed and its tables copied in the order of its context's stream, which is non-blocking: the
legacy default stream may have any amount of work queued when a runner is created and first used."""
import os
import re

import numpy as np
import pytest

from oracle import pipelines as PL

gpu = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCES = [os.path.join(ROOT, "ai-gamer_b200", d, f) for d in ("csrc", "host") for f in sorted(os.listdir(os.path.join(ROOT, "ai-gamer_b200", d)))
           if f.endswith((".cu", ".cuh", ".cpp", ".h"))]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_no_fill_or_copy_on_the_legacy_stream(path):
    """Kernels and runners name a stream in every fill and copy.  (host/layers/ is bound to the legacy stream like the
    reference's classes and waits for it after each of its own.)"""
    text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(path).read(), flags=re.S)
    assert re.findall(r"\bcudaMem(?:set|cpy|cpy2D|set2D|cpyToSymbol|cpyFromSymbol)\s*\(", text) == []


@pytest.fixture(scope="module")
def env():
    import torch
    from tests import gpu_util as U

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    U.ctx()   # (torch leaves the legacy stream)
    return U


def _clips(U, pk, ctx):
    from ai_gamer_b200 import runners as R

    x = U.dev(PL.make_clips(4, 2, 4, 33, 62))
    blob = PL.serialize_conv3d_params(PL.make_conv3d_params(3, trivial=False))

    def make():
        r = R.ClipEncoder(ctx, 2, 4, 33, 62)
        r.load_bytes(blob)
        r.forward(x)
        return r, lambda: (r.outputs_f32(), r.features())
    return make


def _frames(U, pk, ctx, B):
    widths, H, W = (32, 64, 128, 256), 70, 90
    x = U.dev(PL.make_frames(5, B, H, W))
    blob = PL.serialize_cnn_checkpoint(PL.make_cnn_params(1, widths=widths, trivial=False), W, H)

    def make():
        r = pk.CnnEncoder(ctx, B, H, W, widths=widths)
        r.load_bytes(blob)
        r.forward(x)
        return r, lambda: (r.outputs_f32(), r.features())
    return make


def _step(U, pk, ctx):
    from ai_gamer_b200 import runners as R

    x = U.dev(PL.make_embeddings(5, 1, 3, 128)[0])
    blob = PL.serialize_seq_params(PL.make_seq_params(5, d=128, hid=128, layers=2, heads=2))

    def make():
        r = R.SeqHead(ctx, 3, 16, in_c=128, hidden=128, layers=2, heads=2, window=16)
        r.load_bytes(blob)
        r.step(x)
        return r, lambda: (r.outputs_f32(step=True), r.lstm_output(step=True))
    return make


@gpu
@pytest.mark.parametrize("kind", ["clips", "frames_chain", "frames_by_rows", "step"])
def test_runner_made_while_the_legacy_stream_is_busy(env, monkeypatch, kind):
    U = env
    import torch

    pk = U.pkg()
    monkeypatch.setenv("AIG_CNN_NO_CHAIN", "1" if kind == "frames_by_rows" else "0")
    ctx = pk.Context(0, use_torch_stream=False)   # the stream that a context makes itself
    make = {"clips": _clips, "frames_chain": lambda *a: _frames(*a, 2), "frames_by_rows": lambda *a: _frames(*a, 3), "step": _step}[kind](U, pk, ctx)
    first, out = make()
    ctx.sync()
    want = [U.host(t).copy() for t in out()]
    assert all(np.isfinite(w.astype(np.float32)).all() for w in want)
    first.close()
    dirt = torch.full((256 << 20,), 0x7E, dtype=torch.uint8, device="cuda")   # as fp16: NaN
    torch.cuda.synchronize()
    del dirt
    torch.cuda.empty_cache()
    with torch.cuda.stream(torch.cuda.default_stream()):
        torch.cuda._sleep(200_000_000)            # about a tenth of a second, far longer than all below
    second, out = make()
    ctx.sync()
    got = [U.host(t).copy() for t in out()]
    torch.cuda.synchronize()
    late = [U.host(t).copy() for t in out()]      # nothing lands on them afterwards
    for w, g, l in zip(want, got, late):
        assert np.array_equal(w, g) and np.array_equal(w, l)
    second.close()
    ctx.close()
