"""GPU parity of the host-side runners for the sequence head (LSTM -> MHA -> LayerNorm -> FC) and
the streaming agent (frame encoder -> FC -> sequence-head step with carried state and ring cache)
against the oracle compositions.  Streaming must reproduce the full-sequence forward step by step."""
import numpy as np
import pytest

from oracle import oracle as O
from oracle import pipelines as PL

gpu = pytest.mark.gpu
TOL = 2e-2  # relative tolerance on the outputs (fp16 compute)


@pytest.fixture(scope="module")
def env():
    import torch
    from tests import gpu_util as U

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return U


def _seq_head(U, batch, seq_len, d, heads, window):
    from ai_gamer_b200 import runners as R

    return R.SeqHead(U.ctx(), batch, seq_len, in_c=d, hidden=d, layers=2, heads=heads, rope_base=10000.0, window=window)


@gpu
@pytest.mark.parametrize("B,unfused", [(4, "0"), (6, "0"), (1, "0"), (6, "1")])   # the one-kernel step, and the launches per operator
def test_sequence_head_full_and_streaming(env, monkeypatch, B, unfused):
    U = env
    monkeypatch.setenv("AIG_SEQ_NO_FUSED_STEP", unfused)
    U.pkg()
    T, d, heads = 16, 128, 2
    p = PL.make_seq_params(5, d=d, hid=d, layers=2, heads=heads)
    emb = PL.make_embeddings(5, T, B, d)                    # [T][B][d]
    y, a, logits, want = PL.seq_forward(p, emb, rope_base=10000.0, window=0)
    head = _seq_head(U, B, T, d, heads, 0)
    blob = PL.serialize_seq_params(p)
    assert len(blob) == head.param_bytes()
    head.load_bytes(blob)
    emb_bt = np.ascontiguousarray(emb.transpose(1, 0, 2))    # the runner is batch-major
    head.forward(U.dev(emb_bt))
    got_y = U.host(head.lstm_output())
    assert np.abs(got_y.astype(np.float32) - y.transpose(1, 0, 2).astype(np.float32)).max() < 6e-3
    got = U.host(head.outputs_f32())
    assert U.rel_err(got, want.astype(np.float32), 0.05).max() < TOL
    # streaming: the same sequence one frame at a time
    outs = []
    for t in range(T):
        head.step(U.dev(np.ascontiguousarray(emb[t])))
        outs.append(U.host(head.outputs_f32(step=True)))
    got_s = np.stack(outs, axis=1)
    assert U.rel_err(got_s, want.astype(np.float32), 0.05).max() < TOL
    assert np.abs(got_s - got).max() < 5e-3, "streaming and full-sequence forward disagree"
    # reset starts a new sequence
    head.reset()
    head.step(U.dev(np.ascontiguousarray(emb[0])))
    assert np.abs(U.host(head.outputs_f32(step=True)) - got_s[:, 0]).max() < 1e-6
    head.close()


@gpu
def test_streaming_agent_matches_oracle(env):
    U = env
    import torch

    U.pkg()
    from ai_gamer_b200 import runners as R

    B, H, W, widths, d, heads, window, steps = 2, 32, 64, (32, 64), 128, 2, 8, 12
    p = PL.make_agent_params(3, widths=widths, d=d, layers=2, heads=heads)
    frames = [PL.make_frames(100 + t, B, H, W) for t in range(steps)]
    emb = np.stack([O.fc(PL.cnn_forward(p["cnn"], f)[0], p["bw"], p["bb"]) for f in frames])   # [T][B][d]
    _, _, _, want = PL.seq_forward(p["seq"], emb, rope_base=10000.0, window=window)             # [B][T][n_out]
    agent = R.Agent(U.ctx(), B, H, W, widths=widths, d=d, layers=2, heads=heads, window=window)
    blob = PL.serialize_agent_params(p, W, H)
    assert len(blob) == agent.param_bytes()
    agent.load_bytes(blob)
    outs = []
    for t in range(steps):
        agent.step(U.dev(frames[t]))
        outs.append(U.host(agent.outputs_f32()))
    got = np.stack(outs, axis=1)
    assert U.rel_err(got, want.astype(np.float32), 0.05).max() < TOL
    # the host-buffer frame step returns the same numbers
    agent.reset()
    out_h = torch.empty((B, 18), dtype=torch.float32).pin_memory()
    for t in range(3):
        agent.step_host(torch.from_numpy(frames[t]).pin_memory(), out_h)
        assert np.array_equal(out_h.numpy(), got[:, t])
    agent.close()


@gpu
def test_clip_encoder_matches_oracle(env):
    """Conv3D temporal encoder (three Conv3D+BN+LeakyReLU layers, 2x2 adaptive pool, FC head) on short
    clips against the oracle composition, with non-trivial BatchNorm statistics and biases."""
    U = env
    U.pkg()
    from ai_gamer_b200 import runners as R

    B, D, H, W = 2, 4, 32, 64
    p = PL.make_conv3d_params(7, trivial=False)
    clips = PL.make_clips(7, B, D, H, W)
    feat, logits, want = PL.conv3d_forward(p, clips)
    enc = R.ClipEncoder(U.ctx(), B, D, H, W)
    blob = PL.serialize_conv3d_params(p)
    assert len(blob) == enc.param_bytes()
    enc.load_bytes(blob)
    enc.forward(U.dev(clips))
    got_feat = U.host(enc.features()).astype(np.float32)
    assert U.scaled_err(got_feat, feat.astype(np.float32)) < 1e-2
    got = U.host(enc.outputs_f32())
    assert U.rel_err(got, want.astype(np.float32), 0.05).max() < TOL
    # a second call on the same buffers is deterministic
    enc.forward(U.dev(clips))
    assert np.array_equal(U.host(enc.outputs_f32()), got)
    with pytest.raises(Exception, match="size"):
        enc.load_bytes(blob[:-2])                            # a short blob is refused before anything is copied
    enc.close()


@gpu
@pytest.mark.parametrize("rows", [32, 64])
def test_fc_layernorm_swish_twin(env, rows):
    """The CPU-runnable configuration's GPU twin: FC 1024->1024, row LayerNorm (eps 1e-5), Swish; 64 rows is the
    configuration's own batch."""
    U = env
    pk = U.pkg()
    import torch

    c = U.ctx()
    d = 1024
    p = PL.make_fc_ln_params(11, d, d)
    x = np.random.default_rng(11).standard_normal((rows, d)).astype(np.float16)
    want = PL.fc_ln_swish_forward(p, x)
    plan = pk.FcPlan(c, rows, d, d, two_step=True)
    dW, db, dg, dbeta, dx = (U.dev(a) for a in (p["W"], p["b"], p["gamma"], p["beta"], x))  # kept alive to the sync
    plan.set_weights(dW, db)
    y = torch.empty((rows, d), dtype=torch.float16, device="cuda")
    plan.forward(dx, y)
    z = torch.empty_like(y)
    c.call("aig_layernorm_rows_forward", U.p(z), U.p(y), U.p(dg), U.p(dbeta), rows, d, 1e-5)
    c.call("aig_swish_forward", U.p(z), rows * d)
    c.sync()
    got = U.host(z).astype(np.float32)
    assert np.abs(got - want.astype(np.float32)).max() < 6e-3
    assert U.rel_err(got, want.astype(np.float32), 0.05).max() < TOL


@gpu
@pytest.mark.parametrize("B,in_c,d,heads,window,layers", [
    (1, 16, 64, 1, 1, 1), (8, 48, 64, 1, 3, 1), (9, 272, 128, 2, 4, 2), (16, 128, 64, 1, 5, 3), (17, 64, 192, 3, 2, 2), (33, 80, 64, 1, 128, 2),
    (64, 32, 64, 1, 4, 4), (65, 64, 128, 2, 3, 1), (128, 48, 64, 1, 4, 2), (4, 512, 512, 8, 64, 2)])
def test_streaming_step_shapes(env, B, in_c, d, heads, window, layers):
    """The one-kernel step over its range: one sequence to 128 (full and ragged tiles of eight, one and two tiles a warp,
    one to eight warps along K), input widths that leave half a block of K, windows that wrap, one to four layers."""
    U = env
    U.pkg()
    from ai_gamer_b200 import runners as R

    T = 6
    p = PL.make_seq_params(B + d, d=in_c, hid=d, layers=layers, heads=heads)
    emb = PL.make_embeddings(3, T, B, in_c)
    _, _, _, want = PL.seq_forward(p, emb, rope_base=10000.0, window=window)
    head = R.SeqHead(U.ctx(), B, 16, in_c=in_c, hidden=d, layers=layers, heads=heads, rope_base=10000.0, window=window)
    head.load_bytes(PL.serialize_seq_params(p))
    for run in range(2):
        outs = []
        for t in range(T):
            head.step(U.dev(np.ascontiguousarray(emb[t])))
            outs.append(U.host(head.outputs_f32(step=True)))
        got = np.stack(outs, axis=1)
        assert U.rel_err(got, want.astype(np.float32), 0.2).max() < TOL   # an output near zero: 4e-3 absolute
        head.reset()
    head.close()


@gpu
@pytest.mark.parametrize("B,T,d,heads,n_out", [(1, 3, 64, 1, 1), (2, 7, 192, 3, 31), (1, 65, 512, 8, 32), (3, 128, 128, 2, 18), (3, 5, 128, 2, 40)])
def test_whole_sequences_tail_shapes(env, B, T, d, heads, n_out):
    """LayerNorm, FC and activations in one launch: ragged groups of 16 rows, one column tile to four, more outputs than
    it takes; widths of two to sixteen blocks of 32; attention tiles of 64 and 128 keys."""
    U = env
    U.pkg()
    from ai_gamer_b200 import runners as R

    p = PL.make_seq_params(B + n_out, d=d, hid=d, layers=1, heads=heads, n_out=n_out)
    emb = PL.make_embeddings(9, T, B, d)
    n_sig = n_out - n_out // 3
    _, _, _, want = PL.seq_forward(p, emb, rope_base=10000.0, n_sigmoid=n_sig)
    head = R.SeqHead(U.ctx(), B, T, in_c=d, hidden=d, layers=1, heads=heads, n_out=n_out, n_sigmoid=n_sig, rope_base=10000.0)
    head.load_bytes(PL.serialize_seq_params(p))
    dev = U.dev(np.ascontiguousarray(emb.transpose(1, 0, 2)))
    head.forward(dev, 5)
    other = U.host(head.outputs_f32())
    head.forward(dev)
    got = U.host(head.outputs_f32())
    assert U.rel_err(got, want.astype(np.float32), 0.2).max() < TOL
    assert np.abs(other - got).max() < 8e-3   # rotary attention depends on distances only; the angles round differently
    head.close()


def _nontrivial_agent_params(seed, widths, d, heads):
    p = PL.make_agent_params(seed, widths=widths, d=d, layers=2, heads=heads)
    p["cnn"] = PL.make_cnn_params(seed, widths=widths, trivial=False)   # scale and shift that differ from load to load
    return p


@gpu
@pytest.mark.parametrize("B,unfused", [(2, "0"), (6, "0"), (2, "1")])   # step as one captured graph, and as the encoder's graph and launches of its own
def test_agent_second_parameter_load(env, monkeypatch, B, unfused):
    """Parameters loaded a second time take effect in full on input buffers that have been used before."""
    U = env
    import torch

    U.pkg()
    from ai_gamer_b200 import runners as R

    monkeypatch.setenv("AIG_SEQ_NO_FUSED_STEP", unfused)
    H, W, widths, d, heads, window = 32, 64, (32, 64), 128, 2, 8
    blobs = [PL.serialize_agent_params(_nontrivial_agent_params(s, widths, d, heads), W, H) for s in (3, 4)]
    frames = PL.make_frames(9, B, H, W)
    dev, pinned = U.dev(frames), torch.from_numpy(frames).pin_memory()

    def run(agent):
        agent.reset()
        agent.step(dev)
        a = U.host(agent.outputs_f32()).copy()
        out = torch.empty((B, 18), dtype=torch.float32).pin_memory()
        agent.step_host(pinned, out)
        return a, out.numpy().copy()

    def make():
        return R.Agent(U.ctx(), B, H, W, widths=widths, d=d, layers=2, heads=heads, window=window)

    want = []
    for blob in blobs:
        fresh = make()
        fresh.load_bytes(blob)
        want.append(run(fresh))
        fresh.close()
    assert not np.array_equal(want[0][0], want[1][0])
    agent = make()
    for i in (0, 1, 0):
        agent.load_bytes(blobs[i])
        for got, w in zip(run(agent), want[i]):
            assert np.array_equal(got, w), "load of blob %d" % i
    agent.close()


@gpu
@pytest.mark.parametrize("B,D,H,W,offset,widths", [
    (1, 1, 12, 16, 0, (3, 32, 64, 128)),       # a clip of one frame: only the middle depth tap
    (3, 5, 37, 53, 0, (3, 32, 64, 128)),       # odd extents in every layer, tiles that span clips
    (1, 11, 33, 66, 0, (3, 32, 64, 128)),      # more depths than accumulators
    (5, 2, 18, 31, 4, (3, 32, 64, 128)),       # first layer by the gather (clips off a 16-byte boundary)
    (1, 3, 17, 300, 0, (3, 32, 64, 128)),      # and by rows beyond 256 pixels
    (16, 8, 70, 90, 0, (3, 32, 64, 128)),      # several tiles a CTA, runs that begin and end inside a tile
    (2, 4, 40, 48, 0, (3, 32, 128, 32)),       # two channel shares, then a layer that the walk does not take
    (2, 4, 40, 48, 0, (3, 32, 64, 32)),        # one share of 32 channels
])
def test_clip_encoder_depth_walk(env, B, D, H, W, offset, widths):
    """The depth-walking 3-D convolution at the edges of its tiles, runs and channel shares: every layer's output against the
    oracle's, and the same bits from one forward to the next."""
    U = env
    U.pkg()
    import torch
    from ai_gamer_b200 import runners as R

    p = PL.make_conv3d_params(B + D, widths=widths, trivial=False)
    clips = PL.make_clips(W, B, D, H, W)
    enc = R.ClipEncoder(U.ctx(), B, D, H, W, widths=widths)
    assert enc.walked_layers == (1 if widths == (3, 32, 128, 32) else 2)
    enc.load_bytes(PL.serialize_conv3d_params(p))
    room = torch.zeros(clips.size + 8, dtype=torch.float16, device="cuda")
    room[offset:offset + clips.size] = U.dev(clips).flatten()
    torch.cuda.synchronize()
    runs = []
    for _ in range(3):
        enc.forward(room[offset:])
        runs.append([U.host(enc.features())] + [U.host(enc.stage_output(i)) for i in range(len(widths) - 1)])
    assert all(np.array_equal(x, y) for r in runs[1:] for x, y in zip(runs[0], r))
    x = clips
    for i, L in enumerate(p["layers"]):
        x = O.leaky_relu(O.batchnorm(O.conv3d(x, L["w"], L["b"], 1, 2, 1, 1), *L["bn"]), 0.01)
        # element by element, against a scale of at least the rms: the oracle rounds to fp16 after the convolution, BatchNorm
        # and activation, this once a layer (2^-11 each, up to three times the value where BatchNorm shifts it), and each
        # layer carries on what the ones before it differ by
        err = U.scaled_err(runs[0][1 + i], np.moveaxis(x, 1, -1))
        assert err < (i + 1) * 4e-3, "layer %d: %.5f" % (i, err)
    # and the pool, whose mean takes the roundings out again, adds its own
    feat = O.adaptive_avgpool3d(x, 2, 2).astype(np.float32)
    assert U.scaled_err(runs[0][0].astype(np.float32).reshape(feat.shape), feat) < 4e-3
    enc.close()


@gpu
def test_clip_encoder_depth_walk_keeps_infinities_in_their_windows(env):
    """An infinity and a NaN in two clips: the features that their windows reach are as finite as the oracle's, the other
    clips keep their bits, and so does the next forward."""
    U = env
    U.pkg()
    from ai_gamer_b200 import runners as R

    B, D, H, W = 5, 6, 72, 104
    p = PL.make_conv3d_params(9, trivial=False)
    clips = PL.make_clips(9, B, D, H, W)
    bad = clips.copy()
    bad[1, 0, 5, 10, 12] = np.inf       # in the first of the four cells
    bad[3, 2, 0, 60, 90] = np.nan       # in the last
    enc = R.ClipEncoder(U.ctx(), B, D, H, W)
    assert enc.walked_layers == 2
    enc.load_bytes(PL.serialize_conv3d_params(p))

    def run(x):
        enc.forward(U.dev(x))
        return U.host(enc.features()), U.host(enc.outputs_f32())

    clean, dirty = run(clips), run(bad)
    assert all(np.isfinite(a.astype(np.float32)).all() for a in clean)
    want = np.isfinite(PL.conv3d_forward(p, bad)[0].astype(np.float32)).reshape(B, -1)
    assert 0 < (~want[1]).sum() < want[1].size and 0 < (~want[3]).sum() < want[3].size
    assert np.array_equal(np.isfinite(dirty[0].astype(np.float32)).reshape(B, -1), want)
    for d, k in zip(dirty, clean):
        assert np.array_equal(d[[0, 2, 4]], k[[0, 2, 4]])
    assert np.array_equal(dirty[0].reshape(B, -1)[want], clean[0].reshape(B, -1)[want])
    assert all(np.array_equal(a, b) for a, b in zip(run(clips), clean))
    enc.close()
