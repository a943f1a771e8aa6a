"""End-to-end GPU parity of the 2-D frame encoder (host runner + kernels) against the oracle
composition, on the benchmark configuration's shapes at a batch the oracle finishes in seconds."""
import numpy as np
import pytest

from oracle import oracle as O
from oracle import pipelines as PL

gpu = pytest.mark.gpu

REL_TOL = 2e-2    # relative tolerance on the key/mouse outputs (fp16 compute, fp32 accumulation)
STAGE_TOL = 1e-2  # intermediate activations: max error relative to max(|value|, rms of the tensor)


@pytest.fixture(scope="module")
def env():
    import torch
    from tests import gpu_util as U

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return U


@gpu
@pytest.mark.parametrize("trivial", [True, False])
def test_cnn_encoder_matches_oracle(env, trivial):
    U = env
    import torch

    c = U.ctx()
    pk = U.pkg()
    B, H, W = 4, 144, 256
    widths = (32, 64, 128, 256, 256)
    params = PL.make_cnn_params(0 if trivial else 1, widths=widths, trivial=trivial)
    frames = PL.make_frames(0, B, H, W)
    feat, logits, want, stages = PL.cnn_forward(params, frames, return_all=True)
    enc = pk.CnnEncoder(c, B, H, W, widths=widths)
    blob = PL.serialize_cnn_checkpoint(params, W, H)
    assert len(blob) == enc.checkpoint_bytes()
    enc.load_bytes(blob)
    d_frames = U.dev(frames)
    enc.forward(d_frames)
    c.sync()
    # layer by layer first: a failure names the first stage that drifts
    for i, st in enumerate(stages):
        got = U.nchw(U.host(enc.stage_output(i)))
        err = U.scaled_err(got, st)
        assert err < STAGE_TOL, "stage %d: max scaled err %.4f" % (i, err)
    got_feat = U.host(enc.features())
    assert U.rel_err(got_feat, feat, 0.02).max() < REL_TOL
    got = U.host(enc.outputs_f32())
    assert np.array_equal(got.astype(np.float16), U.host(enc.outputs_half()))
    assert U.rel_err(got, want.astype(np.float32), 0.05).max() < REL_TOL
    # decisions (Infer.cpp:8-57): button thresholds must agree wherever the oracle is not within the
    # tolerance of the 0.5 threshold; the mouse deltas (int(p*256)) may differ by one count
    a_got, a_want = O.actions(got, 18, 16), O.actions(want.astype(np.float32), 18, 16)
    clear = np.abs(want.astype(np.float32)[:, :16] - 0.5) > 2e-3
    assert (a_got[:, :16] == a_want[:, :16])[clear].all()
    assert (a_got[:, :16] == a_want[:, :16]).mean() >= 0.999
    assert np.abs(a_got[:, 16:] - a_want[:, 16:]).max() <= 1
    # graph replay and the host-buffer frame step give the same bytes
    enc.forward(d_frames, graph=True)
    c.sync()
    assert np.array_equal(U.host(enc.outputs_f32()), got)
    pinned_in = torch.from_numpy(frames).pin_memory()
    pinned_out = torch.empty((B, 18), dtype=torch.float32).pin_memory()
    enc.infer_host(pinned_in, pinned_out)
    assert np.array_equal(pinned_out.numpy(), got)
    # pipelined submit/wait over two slots: same bytes, any order of slots
    outs = [torch.zeros((B, 18), dtype=torch.float32).pin_memory() for _ in range(2)]
    for step in range(5):
        if step >= 2:
            enc.wait(step & 1)
            assert np.array_equal(outs[step & 1].numpy(), got)
            outs[step & 1].zero_()
        enc.submit_host(step & 1, pinned_in, outs[step & 1])
    for step in (3, 4):
        enc.wait(step & 1)
        assert np.array_equal(outs[step & 1].numpy(), got)
    enc.close()


@gpu
def test_cnn_checkpoint_errors(env):
    U = env
    c = U.ctx()
    pk = U.pkg()
    widths = (32, 64)
    enc = pk.CnnEncoder(c, 1, 32, 64, widths=widths)
    params = PL.make_cnn_params(3, widths=widths)
    blob = PL.serialize_cnn_checkpoint(params, 64, 32)
    with pytest.raises(pk.AigError):
        enc.load_bytes(blob[:-2])  # truncated
    with pytest.raises(pk.AigError):
        enc.load_bytes(PL.serialize_cnn_checkpoint(params, 32, 64))  # wrong resolution in the header
    with pytest.raises(pk.AigError):
        import torch

        enc.forward(torch.zeros(1, dtype=torch.uint8, device="cuda"))  # parameters not loaded
    enc.load_bytes(blob)
    enc.close()


@gpu
def test_full_size_properties(env):
    """The benchmark's own size (256 frames of 144x256) is beyond what the CPU oracle finishes in seconds, so
    the full-size run is checked through properties that do not need it: frames are independent (a frame's
    outputs do not depend on the batch it travels in, up to the fp32 summation order of the tile shape chosen
    for that batch), the run is deterministic bit for bit, the oracle agrees
    on a sample of the frames, and the two convolution paths (fused down-sampling over space-to-depth vs the
    two separate stride-2 convolutions) agree within the fp16 tolerance."""
    U = env
    import os

    c = U.ctx()
    pk = U.pkg()
    B, H, W = 256, 144, 256
    widths = (32, 64, 128, 256, 256)
    params = PL.make_cnn_params(4, widths=widths, trivial=False)
    blob = PL.serialize_cnn_checkpoint(params, W, H)
    frames = PL.make_frames(11, B, H, W)
    enc = pk.CnnEncoder(c, B, H, W, widths=widths)
    enc.load_bytes(blob)
    d_frames = U.dev(frames)
    enc.forward(d_frames)
    c.sync()
    full = U.host(enc.outputs_f32()).copy()
    assert np.isfinite(full).all()
    enc.forward(d_frames)
    c.sync()
    assert np.array_equal(U.host(enc.outputs_f32()), full), "two runs on the same frames differ"
    enc.close()
    # the same frames in batches of 8: other tile shapes (channel-block groups are summed in another order),
    # same values up to a few fp16 ulps; within one batch size the bytes do not depend on the position in the batch
    small = pk.CnnEncoder(c, 8, H, W, widths=widths)
    small.load_bytes(blob)
    for lo in (0, 120, 248):
        small.forward(U.dev(frames[lo:lo + 8]))
        c.sync()
        assert np.abs(U.host(small.outputs_f32()) - full[lo:lo + 8]).max() < 2e-3, "outputs depend on the batch composition"
    small.forward(U.dev(np.ascontiguousarray(frames[7::-1])))
    c.sync()
    rev = U.host(small.outputs_f32()).copy()
    small.forward(U.dev(frames[0:8]))
    c.sync()
    assert np.array_equal(U.host(small.outputs_f32()), rev[::-1]), "a frame's outputs depend on its position in the batch"
    small.close()
    # the oracle on three of the 256 frames
    pick = [0, 131, 255]
    _, _, want = PL.cnn_forward(params, frames[pick])
    assert U.rel_err(full[pick], want.astype(np.float32), 0.05).max() < REL_TOL
    a_got, a_want = O.actions(full[pick], 18, 16), O.actions(want.astype(np.float32), 18, 16)
    clear = np.abs(want.astype(np.float32)[:, :16] - 0.5) > 2e-3
    assert (a_got[:, :16] == a_want[:, :16])[clear].all()
    # the unfused path (two separate stride-2 convolutions per block) on the same frames
    os.environ["AIG_CNN_NO_FUSED_DOWN"] = "1"
    try:
        plain = pk.CnnEncoder(c, B, H, W, widths=widths)
    finally:
        del os.environ["AIG_CNN_NO_FUSED_DOWN"]
    plain.load_bytes(blob)
    plain.forward(d_frames)
    c.sync()
    other = U.host(plain.outputs_f32())
    plain.close()
    assert np.abs(other - full).max() < 4e-3   # outputs live in [-1, 1]


@gpu
def test_recording_file_to_batched_inference(env, tmp_path):
    """Records of the reference's recording format -> planar RGB frames -> batched inference through the pipelined
    host entry point: same outputs as the device path on the BGRA form of the same frames, action agreement with the
    oracle on every record, the last (partial) batch included."""
    U = env
    import struct

    c = U.ctx()
    pk = U.pkg()
    B, H, W, n = 4, 144, 256, 11
    widths = (32, 64, 128, 256, 256)
    params = PL.make_cnn_params(6, widths=widths, trivial=False)
    bgra = PL.make_frames(21, n, H, W)
    planar = np.ascontiguousarray(bgra[..., [2, 1, 0]].transpose(0, 3, 1, 2))          # what the recorder stores
    rng = np.random.default_rng(2)
    keys = rng.integers(0, 1 << 14, n).astype(np.uint16)
    mouse = rng.integers(-200, 200, (n, 2)).astype(np.int32)
    path = tmp_path / "training_data.bin"
    with open(path, "wb") as f:
        f.write(struct.pack("<ii", W, H))
        for i in range(n):
            f.write(struct.pack("<Hii", int(keys[i]), int(mouse[i, 0]), int(mouse[i, 1])))
            f.write(planar[i].tobytes())
    rec = pk.Recording(path)
    assert (rec.width, rec.height, rec.n_records) == (W, H, n)
    enc = pk.CnnEncoder(c, B, H, W, widths=widths)
    enc.load_bytes(PL.serialize_cnn_checkpoint(params, W, H))
    got = rec.infer(enc, 0, n)
    # the device path on BGRA frames, batch by batch
    want_dev = []
    for lo in range(0, n, B):
        chunk = bgra[lo:lo + B]
        if chunk.shape[0] < B:
            chunk = np.concatenate([chunk, np.repeat(chunk[-1:], B - chunk.shape[0], axis=0)])
        enc.forward(U.dev(chunk))
        c.sync()
        want_dev.append(U.host(enc.outputs_f32())[: min(B, n - lo)])
    assert np.array_equal(got, np.concatenate(want_dev)), "planar RGB records and BGRA frames give different outputs"
    # a sub-range
    assert np.array_equal(rec.infer(enc, 3, 5), got[3:8])
    _, _, want = PL.cnn_forward(params, bgra)
    want = want.astype(np.float32)
    assert np.abs(got - want).max() < 2e-3
    a_got, a_want = O.actions(got, 18, 16), O.actions(want, 18, 16)
    clear = np.abs(want[:, :16] - 0.5) > 2e-3
    assert (a_got[:, :16] == a_want[:, :16])[clear].all()
    # the recorded inputs come back as the reference's training targets (Train.cpp:70-76)
    _, k, m = rec.read(0, n)
    t = pk.Recording.targets(k, m)
    assert np.array_equal(t[:, :14], ((keys[:, None] >> np.arange(14)) & 1).astype(np.float32))
    enc.close()
    rec.close()


@gpu
@pytest.mark.parametrize("n", [1, 64, 65, 64 * 9 + 5])
def test_recording_pieces(env, tmp_path, n):
    """Recordings read in pieces by several threads: one frame, one batch, a batch and one frame, and more pieces than
    the pinned ring has slots (56 + 8 frames a batch), against the same frames given to the encoder batch by batch."""
    U = env
    c, pk = U.ctx(), U.pkg()
    B, H, W, widths = 64, 64, 96, (32, 64)
    enc = pk.CnnEncoder(c, B, H, W, widths=widths)
    enc.load_bytes(PL.serialize_cnn_checkpoint(PL.make_cnn_params(7, widths=widths, trivial=False), W, H))
    frames = np.random.default_rng(n).integers(0, 256, (n, 3, H, W), dtype=np.uint8)
    path = tmp_path / "r.bin"
    with open(path, "wb") as f:
        f.write(np.array([W, H], np.int32).tobytes())
        for fr in frames:
            f.write(b"\0" * 10 + fr.tobytes())
    rec = pk.Recording(path)
    got = rec.infer(enc, 0, n)
    for lo in range(0, n, B):
        chunk = np.zeros((B, 3, H, W), np.uint8)
        chunk[: min(B, n - lo)] = frames[lo:lo + B]
        enc.forward_rgb(U.dev(chunk))
        c.sync()
        assert np.array_equal(got[lo:lo + B], U.host(enc.outputs_f32())[: min(B, n - lo)])
    assert np.array_equal(rec.infer(enc, 0, n), got)
    rec.close()
    enc.close()


@gpu
@pytest.mark.parametrize("B,H,W,widths,act", [
    (1, 32, 32, (32, 64), "ACT_SWISH"), (1, 144, 256, (32, 64, 128, 256, 256), "ACT_SWISH"), (3, 67, 131, (32, 64, 128), "ACT_RELU"),
    (6, 120, 200, (32, 64, 128, 256, 256), "ACT_LEAKY"), (19, 107, 189, (32, 64, 128, 256, 256), "ACT_SWISH"), (5, 50, 322, (64, 64, 192), "ACT_SWISH"),
    (150, 20, 20, (32, 64, 128), "ACT_SWISH")])
def test_small_batches_in_one_launch(env, monkeypatch, B, H, W, widths, act):
    """Residual blocks and head as one launch against the per-layer launches: one tile to several rounds of tiles per
    CTA, jobs split over one, two and four CTAs, rows of an image and whole images ending inside a tile, more frames
    than CTAs for the head."""
    U = env
    c, pk = U.ctx(), U.pkg()
    params = PL.make_cnn_params(B + H, widths=widths, trivial=False)
    blob = PL.serialize_cnn_checkpoint(params, W, H)
    frames = U.dev(PL.make_frames(B, B, H, W))
    got = []
    for off in ("1", "0"):
        monkeypatch.setenv("AIG_CNN_NO_CHAIN", off)
        enc = pk.CnnEncoder(c, B, H, W, widths=widths, act=getattr(pk, act))
        enc.load_bytes(blob)
        assert (enc.kernel_launches == 2) == (off == "0")
        runs = []
        for _ in range(3):
            enc.forward(frames)
            c.sync()
            runs.append([U.host(enc.features()), U.host(enc.outputs_f32())] + [U.host(enc.stage_output(i)) for i in range(len(widths))])
        assert all(np.array_equal(x, y) for r in runs[1:] for x, y in zip(runs[0], r))
        got.append([x.astype(np.float32) for x in runs[0]])
        enc.close()
    for i, (a, b) in enumerate(zip(*got)):
        assert U.scaled_err(b, a) < 6e-3, "result %d: %.4f" % (i, U.scaled_err(b, a))   # other summation orders, then a few fp16 roundings


@gpu
@pytest.mark.parametrize("B,chain", [(2, True), (40, False)])
def test_second_parameter_load(env, monkeypatch, B, chain):
    """Parameters loaded a second time take effect in full in graph replays of buffers that have been used before, in
    both frame formats, and in the pipelined host steps."""
    U = env
    import torch

    c, pk = U.ctx(), U.pkg()
    monkeypatch.setenv("AIG_CNN_NO_CHAIN", "0" if chain else "1")
    H, W, widths = 32, 64, (32, 64, 128)
    blobs = [PL.serialize_cnn_checkpoint(PL.make_cnn_params(s, widths=widths, trivial=False), W, H) for s in (1, 2)]
    frames = PL.make_frames(5, B, H, W)
    d_bgra = U.dev(frames)
    d_rgb = U.dev(np.ascontiguousarray(frames[..., [2, 1, 0]].transpose(0, 3, 1, 2)))
    pinned, out = torch.from_numpy(frames).pin_memory(), torch.empty((B, 18), dtype=torch.float32).pin_memory()
    enc = pk.CnnEncoder(c, B, H, W, widths=widths)
    assert (enc.kernel_launches == 2) == chain
    seen = []
    for blob in (blobs[0], blobs[1], blobs[0]):
        enc.load_bytes(blob)
        enc.forward(d_bgra)
        c.sync()
        want = U.host(enc.outputs_f32()).copy()
        seen.append(want)
        enc.forward(d_bgra, graph=True)
        c.sync()
        assert np.array_equal(U.host(enc.outputs_f32()), want)
        enc.forward_rgb(d_rgb, graph=True)
        c.sync()
        assert np.array_equal(U.host(enc.outputs_f32()), want)
        for slot in (0, 1):
            out.zero_()
            enc.submit_host(slot, pinned, out)
            enc.wait(slot)
            assert np.array_equal(out.numpy(), want)
    assert np.array_equal(seen[0], seen[2]) and not np.array_equal(seen[0], seen[1])
    enc.close()


@gpu
@pytest.mark.parametrize("B,H,W,widths", [(2, 48, 80, (32, 64, 128)), (300, 32, 64, (32, 64))])
def test_profile_times_the_launches_of_a_forward(env, B, H, W, widths):
    """Per-launch timing covers the launches that a forward makes, in one launch for the residual blocks or one each, and
    leaves the results as they are."""
    U = env
    c, pk = U.ctx(), U.pkg()
    enc = pk.CnnEncoder(c, B, H, W, widths=widths)
    enc.load_bytes(PL.serialize_cnn_checkpoint(PL.make_cnn_params(8, widths=widths, trivial=False), W, H))
    frames = U.dev(PL.make_frames(3, B, H, W))
    enc.forward(frames)
    c.sync()
    want = U.host(enc.outputs_f32()).copy()
    enc.profile_begin(4)
    for _ in range(4):
        enc.forward(frames)
        c.sync()
        assert np.array_equal(U.host(enc.outputs_f32()), want)
    sites, steps = enc.profile_end()
    assert steps == 4 and len(sites) == enc.kernel_launches and all(0.0 < ms < 50.0 for _, ms, _, _ in sites)
    h, w = (H + 1) // 2, (W + 1) // 2
    flops = 2.0 * B * h * w * widths[0] * 75
    for ci, co in zip(widths, widths[1:]):
        h, w = h // 2, w // 2
        flops += 2.0 * B * h * w * co * (ci * 20 + co * 9)
    flops += 2.0 * B * widths[-1] * 18
    assert abs(sum(f for _, _, f, _ in sites) / flops - 1.0) < 1e-9
    enc.close()


@gpu
def test_checkpoint_files(env, tmp_path):
    """A checkpoint from a file; a file of another size, a directory and a missing file are errors, not exceptions."""
    U = env
    c, pk = U.ctx(), U.pkg()
    enc = pk.CnnEncoder(c, 1, 32, 64, widths=(32, 64))
    blob = PL.serialize_cnn_checkpoint(PL.make_cnn_params(3, widths=(32, 64)), 64, 32)
    (tmp_path / "whole").write_bytes(blob)
    (tmp_path / "short").write_bytes(blob[:-2])
    for name, text in (("short", "does not match"), (".", "does not match"), ("missing", "cannot open")):
        with pytest.raises(pk.AigError, match=text):
            enc.load_file(str(tmp_path / name))
    enc.load_file(str(tmp_path / "whole"))
    enc.forward(U.dev(PL.make_frames(1, 1, 32, 64)))
    c.sync()
    enc.close()


@gpu
@pytest.mark.parametrize("B,H,W,widths,act,walked", [
    (1950, 32, 40, (32, 64, 128), "ACT_SWISH", 4),       # runs of one to eight rows, all the ways they follow one another in the accumulators
    (3, 10, 12, (32, 64, 128), "ACT_RELU", 2),           # one tile, fewer rows than accumulators
    (37, 67, 131, (32, 64, 128, 256), "ACT_LEAKY", 5),   # odd extents, a block by rows before one by patches
    (5, 50, 322, (32, 64, 192), "ACT_SWISH", 2),         # rows beyond 256 pixels; one block by rows
    (150, 20, 20, (32, 64), "ACT_NONE", 2),              # the last block by rows
    (11, 90, 131, (32, 64, 128, 256, 256), "ACT_SWISH", 6),  # 256 channels: whole image rows in a tile, the last one ragged
    (40, 34, 36, (64, 256), "ACT_RELU", 1),              # and into the head directly
    (3, 40, 262, (32, 256, 256), "ACT_LEAKY", 2),        # and a block of them before a block by patches, long rows
])
def test_residual_blocks_by_rows(env, monkeypatch, B, H, W, widths, act, walked):
    """The row-walking residual blocks at the edges of their tiles and runs, every stage against the oracle on a sample.
    `walked`: launches of that kernel."""
    U = env
    c, pk = U.ctx(), U.pkg()
    monkeypatch.setenv("AIG_CNN_NO_CHAIN", "1")
    params = PL.make_cnn_params(B + H, widths=widths, trivial=False)
    frames = PL.make_frames(B, B, H, W)
    pick = np.unique(np.linspace(0, B - 1, 60).astype(int))
    enc = pk.CnnEncoder(c, B, H, W, widths=widths, act=getattr(pk, act))
    assert enc.walked_launches == walked
    enc.load_bytes(PL.serialize_cnn_checkpoint(params, W, H))
    runs = []
    for _ in range(3):
        enc.forward(U.dev(frames))
        c.sync()
        runs.append([U.host(enc.stage_output(i)) for i in range(len(widths))])
    assert all(np.array_equal(x, y) for r in runs[1:] for x, y in zip(runs[0], r))
    stages = PL.cnn_forward(params, frames[pick], act=getattr(O, act), return_all=True)[3]
    for i, (got, want) in enumerate(zip(runs[0], stages)):
        err = U.scaled_err(U.nchw(got[pick]), want)
        assert err < STAGE_TOL, "stage %d: max scaled err %.4f" % (i, err)
    enc.close()


@gpu
@pytest.mark.parametrize("B,H,W,walked", [
    (192, 144, 256, 6), (222, 144, 256, 5), (256, 144, 256, 6), (334, 144, 256, 5),  # rows per CTA against rounds of tiles by patches
    (16, 480, 854, 6), (32, 480, 854, 5),
    (16, 576, 1024, 1), (8, 720, 1280, 1), (8, 380, 672, 5),                        # rows of 65, 81 and twice 43 positions in a tile of 128
    (64, 72, 1392, 2), (64, 72, 1376, 1),                                           # the least that are taken (0.688) and the most that are not (0.680)
    (1, 1400, 400, 5), (1, 576, 1024, 2),                                           # few rows to a tile, many and few rows to a CTA
])
def test_which_convolutions_go_by_rows(env, monkeypatch, B, H, W, walked):
    """256-channel convolutions stay with the patch-resident kernel where that was measured to be the faster one.  (Frames
    of 1024 columns and more have no block by rows, the last block's convolution has half the width.)"""
    U = env
    monkeypatch.setenv("AIG_CNN_NO_CHAIN", "1")
    enc = U.pkg().CnnEncoder(U.ctx(), B, H, W, widths=(32, 64, 128, 256, 256))
    assert enc.walked_launches == walked
    enc.close()


@gpu
def test_blocks_by_rows_keep_infinities_in_their_windows(env, monkeypatch):
    """Activations beyond fp16's range around one bright spot of one image: only what its windows cover becomes infinite
    or NaN, all else keeps its bits, and so does the next forward (the kernel adds to columns that its last tile left)."""
    U = env
    c, pk = U.ctx(), U.pkg()
    monkeypatch.setenv("AIG_CNN_NO_CHAIN", "1")
    B, H, W, widths = 9, 150, 190, (32, 64, 128, 256, 256)
    params = PL.make_cnn_params(4, widths=widths, trivial=False)
    params["c0w"] = (params["c0w"].astype(np.float32) * 4e4).astype(np.float16)   # 255 overflows behind it, 0 and 1 do not
    frames = np.random.default_rng(4).integers(0, 2, (B, H, W, 4), dtype=np.uint8)
    spot = frames.copy()
    image, rows, cols = 4, (70, 73), (90, 93)
    spot[image, rows[0]:rows[1] + 1, cols[0]:cols[1] + 1] = 255
    enc = pk.CnnEncoder(c, B, H, W, widths=widths)
    assert enc.walked_launches == 6
    enc.load_bytes(PL.serialize_cnn_checkpoint(params, W, H))

    def run(f):
        enc.forward(U.dev(f))
        c.sync()
        return [U.host(enc.stage_output(i)) for i in range(len(widths))] + [U.host(enc.features()), U.host(enc.outputs_f32())]

    clean = run(frames)
    assert all(np.isfinite(a.astype(np.float32)).all() for a in clean)
    dirty = run(spot)
    box = [rows, cols]
    for i in range(len(widths)):
        # k5 s2 p2, then per block k4 s2 p1 (the shortcut's window lies inside it) and k3 s1 p1
        box = [((a - 1) // 2, (b + 2) // 2) for a, b in box] if i == 0 else [((a - 1) // 2 - 1, (b + 1) // 2 + 1) for a, b in box]
        inside = np.zeros(clean[i].shape[:3], bool)
        inside[image, max(box[0][0], 0):box[0][1] + 1, max(box[1][0], 0):box[1][1] + 1] = True
        assert not inside.all() and np.array_equal(dirty[i][~inside], clean[i][~inside]), "stage %d" % i
        assert not np.isfinite(dirty[i][inside].astype(np.float32)).all(), "stage %d" % i
    others = np.arange(B) != image
    assert all(np.array_equal(d[others], k[others]) for d, k in zip(dirty[len(widths):], clean[len(widths):]))
    assert all(np.array_equal(a, b) for a, b in zip(run(frames), clean))
    enc.close()
