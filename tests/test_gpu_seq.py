"""GPU parity of the sequence operators (LSTM, multi-head attention with RoPE and the ring KV cache)
through the C ABI against the CPU oracle.  The reference delegates both to cuDNN and pins nothing:
the oracle's definitions (gate order, blob layout, weight orientation, RoPE) are this library's."""
import numpy as np
import pytest

from oracle import oracle as O
from oracle import pipelines as PL

gpu = pytest.mark.gpu


def h(a):
    return np.asarray(a, np.float32).astype(np.float16)


@pytest.fixture(scope="module")
def env():
    import torch
    from tests import gpu_util as U

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return U


LSTM_CASES = [
    # T, B, in, hid, layers, clip, double_bias
    (6, 3, 64, 64, 1, 5.0, True),
    (8, 20, 32, 128, 2, 5.0, True),
    (5, 130, 64, 64, 2, 0.0, False),     # two batch groups, single bias, no clip
    (16, 128, 512, 512, 2, 5.0, True),   # the sequence-head geometry at a short length
]


@gpu
@pytest.mark.parametrize("T,B,I,H,L,clip,dbl", LSTM_CASES)
def test_lstm_matches_oracle(env, T, B, I, H, L, clip, dbl):
    U = env
    import torch

    c = U.ctx()
    pk = U.pkg()
    rng = np.random.default_rng(T * 1000 + B)
    blob = PL.make_lstm_blob(rng, I, H, L, dbl, 1.0)
    if dbl:
        blob[-4 * H:] = h(rng.uniform(-0.2, 0.2, 4 * H))
    x = h(rng.standard_normal((T, B, I)))
    assert blob.size == pk.lib().aig_lstm_weight_count(I, H, L, 1 if dbl else 0)
    want = O.lstm(x, blob, H, L, clip, dbl)
    plan = pk.LstmPlan(c, T, L, H, B, I, clip=clip, double_bias=dbl)
    d_blob = U.dev(blob)
    plan.set_weights(d_blob)
    dy = torch.zeros(T * B * H, dtype=torch.float16, device="cuda")
    plan.forward(U.dev(x), dy)
    c.sync()
    got = U.host(dy).reshape(T, B, H)
    err = np.abs(got.astype(np.float32) - want.astype(np.float32)).max()
    assert err < 6e-3, "max |h - oracle| = %.4g" % err
    # carried state: two halves with state == one pass over the whole sequence
    if T % 2 == 0:
        half = T // 2
        plan2 = pk.LstmPlan(c, half, L, H, B, I, clip=clip, double_bias=dbl)
        plan2.set_weights(d_blob)
        hs = torch.zeros(L * B * H, dtype=torch.float16, device="cuda")
        cs = torch.zeros(L * B * H, dtype=torch.float16, device="cuda")
        y1 = torch.zeros(half * B * H, dtype=torch.float16, device="cuda")
        y2 = torch.zeros(half * B * H, dtype=torch.float16, device="cuda")
        plan2.forward(U.dev(x[:half]), y1, hs, cs, use_state=True)
        plan2.forward(U.dev(x[half:]), y2, hs, cs, use_state=True)
        c.sync()
        both = np.concatenate([U.host(y1), U.host(y2)]).reshape(T, B, H)
        assert np.array_equal(both, got), "streaming halves differ from the full-sequence pass"
        plan2.close()
    plan.close()


@gpu
@pytest.mark.parametrize("T,B,H,L", [
    (1, 1, 64, 2),                                       # a single step, one CTA pair of layers
    (5, 8, 192, 2), (5, 9, 192, 2),                      # half and whole rows delivered; six CTAs in a cluster of eight
    (4, 4, 448, 3), (4, 5, 448, 3),                      # the first and second quad of sequences; a third layer by itself
    (5, 16, 512, 2), (5, 17, 512, 2),                    # W partly in shared memory; a second group
    (4, 48, 512, 2), (4, 49, 512, 2),                    # one group per cluster, two
    (4, 112, 512, 4), (4, 113, 512, 2), (4, 128, 512, 2), (4, 129, 512, 2),  # three and two; beyond: one layer after the other
])
def test_lstm_layers_side_by_side(env, T, B, H, L):
    U = env
    import torch

    c = U.ctx()
    pk = U.pkg()
    rng = np.random.default_rng(B * 1000 + H)
    blob = PL.make_lstm_blob(rng, 32, H, L, True, 1.0)
    blob[-4 * H:] = h(rng.uniform(-0.2, 0.2, 4 * H))
    x = h(rng.standard_normal((T, B, 32)))
    plan = pk.LstmPlan(c, T, L, H, B, 32, clip=5.0, double_bias=True)
    # (how many clusters of 16 CTAs a device holds at once is its own affair, 7 here; six are not too many)
    assert plan.pair_groups == (1, 1) if B <= 48 else plan.pair_groups in ((0, 0), (1, 1), (2, 2), (3, 2))
    plan.set_weights(U.dev(blob))
    dy = torch.zeros(T * B * H, dtype=torch.float16, device="cuda")
    dx = U.dev(x)
    runs = []
    for _ in range(2):  # the counters between the layers are as before after a run
        dy.zero_()
        torch.cuda.synchronize()
        plan.forward(dx, dy)
        c.sync()
        runs.append(U.host(dy).reshape(T, B, H))
    assert np.array_equal(runs[0], runs[1])
    # sequences are independent of each other: the oracle on the first and last ones of the groups
    pick = sorted({0, B - 1, min(B - 1, 15), min(B - 1, 16), min(B - 1, 47), min(B - 1, 48)})
    want = O.lstm(np.ascontiguousarray(x[:, pick]), blob, H, L, 5.0, True)
    # as test_lstm_matches_oracle: fp16 state over a few steps and layers
    assert np.abs(runs[0][:, pick].astype(np.float32) - want.astype(np.float32)).max() < 6e-3
    plan.close()


@gpu
@pytest.mark.parametrize("T,B,H,L,clip,dbl,batch_major", [
    (6, 3, 192, 2, 0.0, False, True),                       # one group a cluster, half of the rows delivered
    (4, 70, 512, 2, 5.0, True, True),                       # two groups, the last one ragged
    (4, 112, 512, 2, 0.0, True, True), (4, 101, 512, 3, 5.0, False, False),   # three and two; a third layer by itself
    (2, 128, 512, 4, 5.0, True, False),                     # two pairs
])
def test_lstm_pairs_with_carried_state(env, T, B, H, L, clip, dbl, batch_major):
    """Two layers in one launch that start from a state and leave one, in both layouts, with and without clip: against the
    oracle, and a sequence in halves against the whole."""
    U = env
    import torch

    c, pk, I = U.ctx(), U.pkg(), 32
    rng = np.random.default_rng(B * 1000 + H + L)
    blob = PL.make_lstm_blob(rng, I, H, L, dbl, 1.0)
    n_bias = 4 * H * L * (2 if dbl else 1)
    blob[-n_bias:] = h(rng.uniform(-0.2, 0.2, n_bias))      # biases of every layer
    x = h(rng.standard_normal((T, B, I)))
    h0, c0 = h(rng.uniform(-1, 1, (L, B, H))), h(rng.standard_normal((L, B, H)))
    order = (1, 0, 2) if batch_major else (0, 1, 2)         # time and sequences change places
    d_blob = U.dev(blob)

    def run(pieces):
        hs, cs, ys = U.dev(h0), U.dev(c0), []
        for piece in pieces:
            t = piece.shape[0]
            plan = pk.LstmPlan(c, t, L, H, B, I, clip=clip, double_bias=dbl, batch_major=batch_major)
            plan.set_weights(d_blob)
            y = torch.zeros(t * B * H, dtype=torch.float16, device="cuda")
            torch.cuda.synchronize()
            plan.forward(U.dev(piece.transpose(order)), y, hs, cs, use_state=True)
            c.sync()
            ys.append(U.host(y).reshape((B, t, H) if batch_major else (t, B, H)).transpose(order))
            plan.close()
        return np.concatenate(ys), U.host(hs), U.host(cs)

    whole = run([x])
    for a, b in zip(whole, run([x[:T // 2], x[T // 2:]])):
        assert np.array_equal(a, b)
    pick = sorted({0, B - 1, min(B - 1, 15), min(B - 1, 16), min(B - 1, 47), min(B - 1, 48), min(B - 1, 64)})
    hw, cw = np.ascontiguousarray(h0[:, pick]), np.ascontiguousarray(c0[:, pick])
    want = O.lstm(np.ascontiguousarray(x[:, pick]), blob, H, L, clip, dbl, hw, cw, True)
    # as test_lstm_matches_oracle for h; the cell state is a sum of a few such steps and up to four times as large
    assert np.abs(whole[0][:, pick].astype(np.float32) - want.astype(np.float32)).max() < 6e-3
    assert np.abs(whole[1][:, pick].astype(np.float32) - hw.astype(np.float32)).max() < 6e-3
    assert np.abs(whole[2][:, pick].astype(np.float32) - cw.astype(np.float32)).max() < 2.4e-2


@gpu
def test_lstm_batch_major_and_step_by_step(env):
    U = env
    import torch

    c = U.ctx()
    pk = U.pkg()
    T, B, I, H, L = 4, 5, 64, 64, 2
    rng = np.random.default_rng(77)
    blob = PL.make_lstm_blob(rng, I, H, L, False, 1.0)
    x = h(rng.standard_normal((T, B, I)))
    want = O.lstm(x, blob, H, L, 0.0, False)
    d_blob = U.dev(blob)
    # cuDNN-8 style layer: batch-major in and out, single bias, no clip (LSTMLayerv8.cpp:9,12,80)
    plan = pk.LstmPlan(c, T, L, H, B, I, clip=0.0, double_bias=False, batch_major=True)
    plan.set_weights(d_blob)
    dy = torch.zeros(B * T * H, dtype=torch.float16, device="cuda")
    plan.forward(U.dev(np.ascontiguousarray(x.transpose(1, 0, 2))), dy)
    c.sync()
    got = U.host(dy).reshape(B, T, H).transpose(1, 0, 2)
    assert np.abs(got.astype(np.float32) - want.astype(np.float32)).max() < 6e-3
    # one step at a time with carried state
    step = pk.LstmPlan(c, 1, L, H, B, I, clip=0.0, double_bias=False)
    step.set_weights(d_blob)
    hs = torch.zeros(L * B * H, dtype=torch.float16, device="cuda")
    cs = torch.zeros(L * B * H, dtype=torch.float16, device="cuda")
    outs = []
    for t in range(T):
        y = torch.zeros(B * H, dtype=torch.float16, device="cuda")
        step.forward(U.dev(x[t:t + 1]), y, hs, cs, use_state=True)
        outs.append(U.host(y).reshape(B, H))
    c.sync()
    assert np.abs(np.stack(outs).astype(np.float32) - want.astype(np.float32)).max() < 6e-3
    plan.close()
    step.close()


@gpu
@pytest.mark.parametrize("B,T,E,Hh,rope,window", [(2, 9, 128, 2, 0.0, 0), (3, 64, 512, 8, 10000.0, 0), (2, 40, 128, 2, 10000.0, 16),
                                                  (2, 100, 128, 2, 10000.0, 0)])
def test_mha_full_sequence(env, B, T, E, Hh, rope, window):
    U = env
    import torch

    c = U.ctx()
    pk = U.pkg()
    rng = np.random.default_rng(B * 100 + T)
    x = h(rng.standard_normal((B, T, E)))
    ws = [PL.xavier_uniform(rng, (E, E), E, E) for _ in range(4)]
    want = O.mha(x, *ws, Hh, rope, 3, window)
    plan = pk.MhaPlan(c, B, T, E, Hh, rope_base=rope, window=window)
    dws = [U.dev(w) for w in ws]
    plan.set_weights(*dws)
    dy = torch.zeros(B * T * E, dtype=torch.float16, device="cuda")
    plan.forward(U.dev(x), dy, pos0=3)
    c.sync()
    got = U.host(dy).reshape(B, T, E)
    assert U.scaled_err(got, want) < 1e-2
    plan.close()


@gpu
def test_mha_streaming_ring_cache_equals_windowed_full_sequence(env):
    U = env
    import torch

    c = U.ctx()
    pk = U.pkg()
    B, E, Hh, window, steps = 2, 128, 2, 8, 21
    rng = np.random.default_rng(9)
    x = h(rng.standard_normal((B, steps, E)))
    ws = [PL.xavier_uniform(rng, (E, E), E, E) for _ in range(4)]
    want = O.mha(x, *ws, Hh, 10000.0, 0, window)  # sliding window of `window` steps
    plan = pk.MhaPlan(c, B, window, E, Hh, rope_base=10000.0, window=window)
    dws = [U.dev(w) for w in ws]
    plan.set_weights(*dws)
    outs = []
    for t in range(steps):
        y = torch.zeros(B * E, dtype=torch.float16, device="cuda")
        plan.step(U.dev(np.ascontiguousarray(x[:, t])), y, t)
        outs.append(U.host(y).reshape(B, E))
    c.sync()
    got = np.stack(outs, axis=1)
    assert U.scaled_err(got, want) < 1e-2
    # after a reset the cache is empty again
    plan.reset()
    y = torch.zeros(B * E, dtype=torch.float16, device="cuda")
    plan.step(U.dev(np.ascontiguousarray(x[:, 0])), y, 0)
    c.sync()
    assert U.scaled_err(U.host(y).reshape(B, E), want[:, 0]) < 1e-2
    plan.close()


@gpu
@pytest.mark.parametrize("T", [16, 100])   # both tile kernels
def test_mha_rotation_beside_a_replayed_capture(env, T):
    """A captured forward of some positions, replayed between eager forwards of others: each call rotates by its own
    positions, whatever ran before it."""
    U = env
    import torch

    c, pk = U.ctx(), U.pkg()
    B, E, Hh = 2, 128, 2
    rng = np.random.default_rng(T)
    plan = pk.MhaPlan(c, B, T, E, Hh, rope_base=10000.0)
    plan.set_weights(*[U.dev(PL.xavier_uniform(rng, (E, E), E, E)) for _ in range(4)])
    x = U.dev(h(rng.standard_normal((B, T, E))))
    y = torch.zeros(B * T * E, dtype=torch.float16, device="cuda")
    yg = torch.zeros_like(y)

    def eager(pos0):
        plan.forward(x, y, pos0=pos0)
        c.sync()
        return U.host(y).copy()

    at = {pos0: eager(pos0) for pos0 in (-1, 0, 5)}
    assert not np.array_equal(at[0], at[5])     # the rounding of the rotated halves differs
    assert np.array_equal(eager(-1), at[-1])    # the plan's first forward had made its table
    c.graph_begin()
    plan.forward(x, yg, pos0=5)
    g = c.graph_end()
    for replays in range(3):
        assert np.array_equal(eager(0), at[0]), "eager forward after %d replays" % replays
        yg.zero_()
        torch.cuda.synchronize()
        c.graph_launch(g)
        c.sync()
        assert np.array_equal(U.host(yg), at[5])
        assert np.array_equal(eager(0), at[0]), "eager forward after a replay"
    pk.lib().aig_graph_destroy(g)
    plan.close()
