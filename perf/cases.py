"""The work a user of this framework has it do, as measurable cases through its public entry points.

Every case has a `kind`:

  agent_host   one frame of the streaming agent with host buffers in and out: the loop body of a player (Agent.step_host)
  agent_step   one frame for each of `batch` concurrent sequences, frames already on the device (Agent.step)
  encoder      a batch of BGRA or planar RGB frames through the 2-D frame encoder (CnnEncoder.forward / forward_rgb)
  clips        a batch of clips through the 3-D convolution clip encoder (ClipEncoder.forward)
  sequences    whole embedding sequences through LSTM, attention, LayerNorm and FC (SeqHead.forward)
  fc_train     one training step of a fully connected layer: forward, loss gradient, backward, AdamW
  refnet       one frame through the reference's own network under the reference's names (aig_refnn_infer_frame)
  recording    offline inference over a recording file (Recording.infer)

Weights and inputs are drawn from the seed with the distributions the benchmark states: He-normal and Xavier weights,
uniform bytes for frames, uniform [0, 1] clips, N(0, 1) embeddings.
"""
import ctypes
import importlib
import math
import os
import tempfile

import numpy as np
import torch

pkg = importlib.import_module("ai-gamer_b200")
runners = importlib.import_module("ai-gamer_b200.runners")
synth = importlib.import_module("ai-gamer_b200.synth")

WIDTHS = (32, 64, 128, 256, 256)   # frame encoder channels
CLIP_WIDTHS = (3, 32, 64, 128)     # clip encoder channels
N_OUT = 18                         # 16 keys and 2 mouse axes
REFNET_OUT = 16


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a live player: one 256x144 frame from the host, actions back on the host, 64 frames of context
        {"name": "agent_host_b1", "kind": "agent_host", "batch": 1, "height": 144, "width": 256, "window": 64},
        # a server stepping 128 players (the per-GPU share of 1024 sequences)
        {"name": "agent_step_b128", "kind": "agent_step", "batch": 128, "height": 144, "width": 256, "window": 64},
        # a handful of players with a frame size of their own
        {"name": "agent_step_b6", "kind": "agent_step", "batch": 6, "height": 120, "width": 200, "window": 64},
        # the frame encoder at the batch its configuration states, replayed as a graph
        {"name": "encoder_b32", "kind": "encoder", "batch": 32, "height": 144, "width": 256, "layout": "bgra", "graph": True},
        # and at the batch of the headline metric
        {"name": "encoder_b256", "kind": "encoder", "batch": 256, "height": 144, "width": 256, "layout": "bgra", "graph": False},
        # frames as a recorder stores them, at an odd size and a ragged batch
        {"name": "encoder_b19_odd", "kind": "encoder", "batch": 19, "height": 107, "width": 189, "layout": "rgb", "graph": False},
        # the temporal configuration: 16 clips of 8 frames
        {"name": "clips_b16", "kind": "clips", "batch": 16, "depth": 8, "height": 144, "width": 256},
        # the sequence head over whole recorded sequences (the prefill of a context)
        {"name": "sequences_b128_t64", "kind": "sequences", "batch": 128, "seq_len": 64, "in_c": 512, "hidden": 512},
        # a short ragged one with a narrower head
        {"name": "sequences_b3_t37", "kind": "sequences", "batch": 3, "seq_len": 37, "in_c": 272, "hidden": 256},
        # a training step of the fully connected layer at the reference's stated shape
        {"name": "fc_train_b64", "kind": "fc_train", "batch": 64, "in_c": 1024, "out_c": 1024},
        # the network a user of the reference brings along, frame by frame
        {"name": "refnet_frame", "kind": "refnet", "height": 144, "width": 256},
        # labelling a recording offline
        {"name": "recording_600", "kind": "recording", "records": 600, "batch": 256, "height": 144, "width": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _frame_size(rng):
    return rng.randint(64, 180), rng.randint(96, 320)


def draw(rng):
    kind = rng.choice(["agent_host", "agent_step", "encoder", "clips", "sequences", "fc_train", "refnet", "recording"])
    if kind in ("agent_host", "agent_step"):
        h, w = _frame_size(rng)
        most = 4 if kind == "agent_host" else max(2, min(128, 128 * 144 * 256 // (h * w)))
        return {"kind": kind, "batch": _log_int(rng, 1 if kind == "agent_host" else 2, most), "height": h, "width": w, "window": rng.choice([16, 32, 64])}
    if kind == "encoder":
        h, w = _frame_size(rng)
        return {"kind": kind, "batch": _log_int(rng, 1, min(256, 256 * 144 * 256 // (h * w))), "height": h, "width": w,
                "layout": rng.choice(["bgra", "rgb"]), "graph": rng.random() < 0.5}
    if kind == "clips":
        h, w = _frame_size(rng)
        depth = rng.randint(4, 12)
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, min(16, 16 * 8 * 144 * 256 // (depth * h * w)))), "depth": depth, "height": h, "width": w}
    if kind == "sequences":
        t = _log_int(rng, 4, 128)
        return {"kind": kind, "batch": _log_int(rng, 1, min(128, 8192 // t)), "seq_len": t, "in_c": 16 * rng.randint(8, 32), "hidden": rng.choice([128, 256, 512])}
    if kind == "fc_train":
        return {"kind": kind, "batch": _log_int(rng, 16, 256), "in_c": 8 * _log_int(rng, 32, 256), "out_c": 2 * _log_int(rng, 8, 512)}
    if kind == "refnet":
        return {"kind": kind, "height": rng.randint(48, 144), "width": rng.randint(64, 256)}
    h, w = _frame_size(rng)
    most = 600 * 144 * 256 // (h * w)
    return {"kind": kind, "records": _log_int(rng, 64, min(600, most)), "batch": rng.choice([32, 64, 128, 256]), "height": h, "width": w}


# ------------------------------------------------------------------------------------------------ states
class _Kept:
    """A runner, plan or handle together with what it needs to be there; closed once nothing refers to it any more."""

    def __init__(self, thing, *needs):
        self.thing, self.needs = thing, needs

    def __del__(self):
        self.thing.close()


class _Buffer:
    """Device memory that a runner owns, as the array interface torch reads; the runner stays as long as the memory is used."""

    def __init__(self, kept, address, shape, typestr):
        self.kept = kept
        self.__cuda_array_interface__ = {"data": (address, False), "shape": tuple(shape), "typestr": typestr, "version": 3}


class _State:
    """What a program holds between calls."""

    def __init__(self, case):
        self.case, self.kept = case, []
        self.ctx = self.own(pkg.Context(0))

    def own(self, thing):
        self.kept.append(_Kept(thing, *self.kept[:1]))
        return thing

    def view(self, thing, address, shape, typestr):
        kept = next(k for k in self.kept if k.thing is thing)
        return torch.as_tensor(_Buffer(kept, address, shape, typestr), device="cuda")


def _generator(seed):
    return torch.Generator("cuda").manual_seed(seed)


def _frames(seed, shape):
    return torch.randint(0, 256, shape, dtype=torch.uint8, device="cuda", generator=_generator(seed))


def _prepare_agent(s, c, seed):
    h, w, b = c["height"], c["width"], c["batch"]
    s.agent = s.own(runners.Agent(s.ctx, b, h, w, widths=WIDTHS, d=512, layers=2, heads=8, n_out=N_OUT, window=c["window"]))
    s.agent.load_bytes(synth.serialize_agent_params(synth.make_agent_params(seed, widths=WIDTHS), w, h))
    host = c["kind"] == "agent_host"
    s.frames = torch.empty((b, h, w, 4), dtype=torch.uint8, device="cpu" if host else "cuda", pin_memory=host)
    if host:
        s.out = torch.empty((b, N_OUT), dtype=torch.float32, pin_memory=True)
        step = lambda: s.agent.step_host(s.frames, s.out)  # noqa: E731
    else:
        s.out = s.view(s.agent, pkg.lib().aig_agent_outputs_f32(s.agent.handle), (b, N_OUT), "<f4")
        step = lambda: s.agent.step(s.frames)  # noqa: E731
    # a running agent: its context window has filled up with earlier frames
    for t in range(c["window"]):
        s.frames.copy_(_frames(1000 * seed + t, s.frames.shape))
        step()
    s.frames.copy_(_frames(1000 * seed + 999, s.frames.shape))


def _prepare_encoder(s, c, seed):
    h, w, b = c["height"], c["width"], c["batch"]
    s.encoder = s.own(pkg.CnnEncoder(s.ctx, b, h, w, widths=WIDTHS, n_out=N_OUT))
    s.encoder.load_bytes(synth.serialize_cnn_checkpoint(synth.make_cnn_params(seed, widths=WIDTHS), w, h))
    s.frames = _frames(seed, (b, h, w, 4) if c["layout"] == "bgra" else (b, 3, h, w))
    s.out = (s.view(s.encoder, pkg.lib().aig_cnn_outputs_f32(s.encoder.handle), (b, N_OUT), "<f4"),
             s.view(s.encoder, pkg.lib().aig_cnn_features(s.encoder.handle), (b, WIDTHS[-1]), "<f2"))


def _prepare_clips(s, c, seed):
    shape = (c["batch"], 3, c["depth"], c["height"], c["width"])
    s.encoder = s.own(runners.ClipEncoder(s.ctx, c["batch"], c["depth"], c["height"], c["width"], widths=CLIP_WIDTHS, n_out=N_OUT))
    s.encoder.load_bytes(synth.serialize_conv3d_params(synth.make_conv3d_params(seed, widths=CLIP_WIDTHS)))
    s.clips = torch.rand(shape, device="cuda", generator=_generator(seed)).half()
    s.out = (s.view(s.encoder, pkg.lib().aig_c3d_outputs_f32(s.encoder.handle), (c["batch"], N_OUT), "<f4"),
             s.view(s.encoder, pkg.lib().aig_c3d_features(s.encoder.handle), (c["batch"], 4 * CLIP_WIDTHS[-1]), "<f2"))


def _prepare_sequences(s, c, seed):
    b, t, d, e = c["batch"], c["seq_len"], c["in_c"], c["hidden"]
    s.head = s.own(runners.SeqHead(s.ctx, b, t, in_c=d, hidden=e, layers=2, heads=e // 64, n_out=N_OUT))
    s.head.load_bytes(synth.serialize_seq_params(synth.make_seq_params(seed, d=d, hid=e, layers=2, heads=e // 64, n_out=N_OUT)))
    s.emb = torch.randn((b, t, d), device="cuda", generator=_generator(seed)).half()
    s.out = (s.view(s.head, pkg.lib().aig_seq_outputs_f32(s.head.handle), (b, t, N_OUT), "<f4"),
             s.view(s.head, pkg.lib().aig_seq_lstm_output(s.head.handle), (b, t, e), "<f2"))


def _prepare_fc_train(s, c, seed):
    b, i, n = c["batch"], c["in_c"], c["out_c"]
    g = _generator(seed)
    half = lambda *shape: torch.zeros(shape, dtype=torch.float16, device="cuda")  # noqa: E731
    s.forward = s.own(pkg.FcPlan(s.ctx, b, i, n, two_step=True))
    s.backward = s.own(pkg.FcBackwardPlan(s.ctx, b, i, n))
    s.x = torch.randn((b, i), device="cuda", generator=g).half()
    s.target = torch.randn((b, n), device="cuda", generator=g).half()
    # the weights live where the layer class keeps them: in the input-gradient GEMM's operand, if its layout allows
    kept = pkg.lib().aig_fc_backward_weight_storage(s.backward.handle)
    s.w = s.view(s.backward, kept, (i, n), "<f2") if kept else half(i, n)
    s.w.copy_(torch.randn((i, n), device="cuda", generator=g) * math.sqrt(2.0 / i))
    s.bias, s.y, s.grad, s.grad_x = half(n), half(b, n), half(b, n), half(b, i)
    s.grad_w, s.grad_b = half(i, n), half(n)
    s.m_w, s.v_w, s.m_b, s.v_b = half(i, n), half(i, n), half(n), half(n)
    s.forward.set_weights(s.w, s.bias)
    s.steps = 0


class _RefNet:
    """The reference's NN class on a handle of the legacy default stream, as its inference loop makes them."""

    def __init__(self, checkpoint):
        lib = pkg.lib()
        self.handle, self.nn = ctypes.c_void_p(), ctypes.c_void_p()
        self._check(lib.aig_compat_handle_create(ctypes.byref(self.handle)))
        fd, path = tempfile.mkstemp(suffix=".ckpt")
        try:
            with os.fdopen(fd, "wb") as f:
                f.write(checkpoint)
            self._check(lib.aig_refnn_create(self.handle, 0, 0, path.encode(), ctypes.byref(self.nn)))
        finally:
            os.unlink(path)

    @staticmethod
    def _check(rc):
        if rc != 0:
            raise pkg.AigError(rc, pkg.lib().aig_layers_last_error().decode())

    def infer_frame(self, bgra, planar, half, out_dev, out_host):
        self._check(pkg.lib().aig_refnn_infer_frame(self.nn, *(pkg.ptr(t) for t in (bgra, planar, half, out_dev, out_host))))

    def close(self):
        pkg.lib().aig_refnn_destroy(self.nn)
        pkg.lib().aig_ctx_destroy(self.handle)


def _prepare_refnet(s, c, seed):
    h, w = c["height"], c["width"]
    s.net = s.own(_RefNet(synth.serialize_refnn_checkpoint(synth.make_refnn_params(seed, w, h))))
    s.bgra = _frames(seed, (h, w, 4))
    s.planar = torch.empty(3 * h * w, dtype=torch.uint8, device="cuda")
    s.half = torch.empty(3 * h * w, dtype=torch.float16, device="cuda")
    s.out_dev = torch.empty(REFNET_OUT, dtype=torch.float32, device="cuda")
    s.out = torch.empty(REFNET_OUT, dtype=torch.float32)


def _prepare_recording(s, c, seed):
    h, w, n = c["height"], c["width"], c["records"]
    s.encoder = s.own(pkg.CnnEncoder(s.ctx, c["batch"], h, w, widths=WIDTHS, n_out=N_OUT))
    s.encoder.load_bytes(synth.serialize_cnn_checkpoint(synth.make_cnn_params(seed, widths=WIDTHS), w, h))
    # width, height, then per record key states, mouse deltas and the planar frame
    records = np.frombuffer(np.random.default_rng(seed).bytes(n * (10 + 3 * h * w)), np.uint8)
    fd, path = tempfile.mkstemp(suffix=".rec")
    try:
        with os.fdopen(fd, "wb") as f:
            f.write(np.array([w, h], np.int32).tobytes())
            f.write(records)
        s.recording = s.own(pkg.Recording(path))
    finally:
        os.unlink(path)   # the recording holds the file open


_PREPARE = {"agent_host": _prepare_agent, "agent_step": _prepare_agent, "encoder": _prepare_encoder, "clips": _prepare_clips,
            "sequences": _prepare_sequences, "fc_train": _prepare_fc_train, "refnet": _prepare_refnet, "recording": _prepare_recording}


def prepare(case, seed):
    s = _State(case)
    _PREPARE[case["kind"]](s, case, seed)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------------------------ one pass
def _run_fc_train(s):
    c = s.case
    s.steps += 1
    s.forward.forward(s.x, s.y)
    s.ctx.call("aig_loss_gradient", pkg.ptr(s.grad), pkg.ptr(s.y), pkg.ptr(s.target), s.y.numel())
    s.backward.backward(s.x, s.grad, s.w, s.grad_w, s.grad_b, s.grad_x)
    s.ctx.call("aig_fc_adamw_update", s.forward.handle, c["in_c"], c["out_c"], *(pkg.ptr(t) for t in (s.w, s.grad_w, s.m_w, s.v_w, s.bias, s.grad_b, s.m_b, s.v_b)),
               1e-4, s.steps, 1e-6)
    return s.y, s.grad, s.grad_x, s.grad_w, s.grad_b, s.w, s.m_w, s.v_w, s.bias, s.m_b, s.v_b


def run(s):
    kind = s.case["kind"]
    if kind == "agent_host":
        s.agent.step_host(s.frames, s.out)
    elif kind == "agent_step":
        s.agent.step(s.frames)
    elif kind == "encoder":
        (s.encoder.forward if s.case["layout"] == "bgra" else s.encoder.forward_rgb)(s.frames, graph=s.case["graph"])
    elif kind == "clips":
        s.encoder.forward(s.clips)
    elif kind == "sequences":
        s.head.forward(s.emb)
    elif kind == "fc_train":
        return _run_fc_train(s)
    elif kind == "refnet":
        s.net.infer_frame(s.bgra, s.planar, s.half, s.out_dev, s.out)
    else:
        return s.recording.infer(s.encoder, 0, s.case["records"])
    return s.out


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _conv(pixels, cin, cout, taps):
    """(operations, weights) of a convolution."""
    return 2.0 * pixels * cin * cout * taps, cin * cout * taps


def _encoder_work(h, w):
    """(operations per frame, weights) of the frame encoder."""
    h, w = (h - 1) // 2 + 1, (w - 1) // 2 + 1
    parts = [_conv(h * w, 3, WIDTHS[0], 25)]
    for i in range(len(WIDTHS) - 1):
        h, w = (h - 2) // 2 + 1, (w - 2) // 2 + 1
        parts += [_conv(h * w, WIDTHS[i], WIDTHS[i + 1], 16 + 4), _conv(h * w, WIDTHS[i + 1], WIDTHS[i + 1], 9)]
    parts.append(_conv(1, WIDTHS[-1], N_OUT, 1))
    return sum(p[0] for p in parts), sum(p[1] for p in parts)


def _clip_work(d, h, w):
    parts = []
    for i in range(len(CLIP_WIDTHS) - 1):
        h, w = (h - 1) // 2 + 1, (w - 1) // 2 + 1
        parts.append(_conv(d * h * w, CLIP_WIDTHS[i], CLIP_WIDTHS[i + 1], 27))
    parts.append(_conv(1, 4 * CLIP_WIDTHS[-1], N_OUT, 1))
    return sum(p[0] for p in parts), sum(p[1] for p in parts)


def _head_work(steps, context, d, e):
    """(operations of `steps` steps with `context` earlier ones each, weights) of the sequence head."""
    weights = 4 * e * (d + e) + 4 * e * (e + e) + 4 * e * e + e * N_OUT
    return steps * (2.0 * weights + 4.0 * context * e), weights


def _refnet_work(h, w):
    h, w = h // 2, w // 2
    parts = [_conv(h * w, 3, 32, 4)]
    for a, b in ((32, 64), (64, 128), (128, 256)):
        h, w = (h - 2) // 2 + 1, (w - 2) // 2 + 1
        parts += [_conv(h * w, a, b, 16 + 4), _conv(h * w, b, b, 9)]
    parts += [_conv(1, 256 * h * w, 1024, 1), _conv(1, 1024, 512, 1), _conv(1, 512, 256, 1), _conv(1, 256, REFNET_OUT, 1)]
    return sum(p[0] for p in parts), sum(p[1] for p in parts)


def work(case):
    c, kind = case, case["kind"]
    if kind in ("agent_host", "agent_step"):
        enc_ops, enc_w = _encoder_work(c["height"], c["width"])
        head_ops, head_w = _head_work(1, c["window"], 512, 512)
        ops = c["batch"] * (enc_ops + head_ops + 2.0 * WIDTHS[-1] * 512)
        frames = c["batch"] * c["height"] * c["width"] * 4
        # the attention cache is read, the recurrent state read and written
        carried = c["batch"] * (2 * c["window"] * 512 * 2 + 2 * 2 * 2 * 512 * 2)
        return {"bytes": frames + 2.0 * (enc_w + head_w + WIDTHS[-1] * 512) + carried + c["batch"] * N_OUT * 4, "flops": ops}
    if kind in ("encoder", "recording"):
        ops, weights = _encoder_work(c["height"], c["width"])
        n = c["batch"] if kind == "encoder" else c["records"]
        pixel = 4 if kind == "encoder" and c["layout"] == "bgra" else 3
        return {"bytes": n * c["height"] * c["width"] * pixel + 2.0 * weights + n * N_OUT * 4 + (n * WIDTHS[-1] * 2 if kind == "encoder" else 0), "flops": n * ops}
    if kind == "clips":
        ops, weights = _clip_work(c["depth"], c["height"], c["width"])
        return {"bytes": c["batch"] * (3 * c["depth"] * c["height"] * c["width"] * 2 + N_OUT * 4 + 4 * CLIP_WIDTHS[-1] * 2) + 2.0 * weights, "flops": c["batch"] * ops}
    if kind == "sequences":
        steps = c["batch"] * c["seq_len"]
        ops, weights = _head_work(steps, (c["seq_len"] + 1) / 2, c["in_c"], c["hidden"])
        return {"bytes": 2.0 * weights + steps * (2 * c["in_c"] + 4 * N_OUT + 2 * c["hidden"]), "flops": ops}
    if kind == "fc_train":
        b, i, n = c["batch"], c["in_c"], c["out_c"]
        # weights and both moments read and written, the gradient written; x, target read; y, its gradient, x's gradient written
        return {"bytes": 2.0 * (7 * (i * n + n) + 2 * b * i + 3 * b * n), "flops": 6.0 * b * i * n}
    ops, weights = _refnet_work(c["height"], c["width"])
    return {"bytes": c["height"] * c["width"] * 4 + 2.0 * weights + REFNET_OUT * 4, "flops": ops}


def tolerance(case):
    # activations are stored as fp16 (2^-11 a rounding) between layers, products summed in fp32: about ten roundings in a row
    if case["kind"] in ("agent_host", "agent_step"):
        return {"rel": 1e-2}   # and 64 steps of carried fp16 state
    if case["kind"] == "sequences":
        return {"rel": 1e-2}   # fp16 state carried over the steps
    if case["kind"] == "fc_train":
        # fp16 moments: a gradient that differs by its last bit moves its weight's step by the same share of it
        return {"rel": 5e-3, "max": 0.5}
    return {"rel": 5e-3}
