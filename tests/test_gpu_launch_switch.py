"""AIG_NO_PDL=1, read when a context is created: every launch of the library follows its predecessor in full.  What a
launch depends on is read off the captured graph's edges, and the results have to be the same bits."""
import ctypes

import numpy as np
import pytest

from oracle import pipelines as PL

gpu = pytest.mark.gpu
PROGRAMMATIC = 1   # CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC


@pytest.fixture(scope="module")
def env():
    import torch
    from tests import gpu_util as U

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return U


def _programmatic_edges(aig_graph):
    """Edges of a captured graph over which a kernel may start before its predecessor has ended."""
    cu = ctypes.CDLL("libcuda.so.1")
    graph = ctypes.cast(aig_graph, ctypes.POINTER(ctypes.c_void_p))[0]   # first member of aig_graph
    n = ctypes.c_size_t()
    assert cu.cuGraphGetEdges_v2(ctypes.c_void_p(graph), None, None, None, ctypes.byref(n)) == 0
    if n.value == 0:
        return 0
    a, b = (ctypes.c_void_p * n.value)(), (ctypes.c_void_p * n.value)()
    data = (ctypes.c_ubyte * (8 * n.value))()   # from_port, to_port, type, five reserved bytes
    assert cu.cuGraphGetEdges_v2(ctypes.c_void_p(graph), a, b, data, ctypes.byref(n)) == 0
    return sum(data[8 * i + 2] == PROGRAMMATIC for i in range(n.value))


def _encoder(U, ctx, B, H, W, widths):
    pk = U.pkg()
    enc = pk.CnnEncoder(ctx, B, H, W, widths=widths)
    enc.load_bytes(PL.serialize_cnn_checkpoint(PL.make_cnn_params(1, widths=widths, trivial=False), W, H))
    frames = U.dev(PL.make_frames(2, B, H, W))
    return enc, lambda: enc.forward(frames), lambda: U.host(enc.outputs_f32()).copy()


def _clips(U, ctx):
    U.pkg()
    from ai_gamer_b200 import runners as R

    enc = R.ClipEncoder(ctx, 2, 4, 32, 64)
    enc.load_bytes(PL.serialize_conv3d_params(PL.make_conv3d_params(3, trivial=False)))
    clips = U.dev(PL.make_clips(4, 2, 4, 32, 64))
    return enc, lambda: enc.forward(clips), lambda: U.host(enc.outputs_f32()).copy()


def _sequences(U, ctx):
    U.pkg()
    from ai_gamer_b200 import runners as R

    head = R.SeqHead(ctx, 3, 16, in_c=128, hidden=128, layers=2, heads=2)
    head.load_bytes(PL.serialize_seq_params(PL.make_seq_params(5, d=128, hid=128, layers=2, heads=2)))
    emb = U.dev(np.ascontiguousarray(PL.make_embeddings(6, 16, 3, 128).transpose(1, 0, 2)))
    return head, lambda: head.forward(emb), lambda: U.host(head.outputs_f32()).copy()


class _FcStep:
    """Forward, loss gradient, backward and AdamW of a fully connected layer, from the same state every time."""

    def __init__(self, U, ctx):
        import torch

        pk = U.pkg()
        self.pk, self.ctx = pk, ctx
        rng = np.random.default_rng(7)
        b, i, n = self.shape = (32, 256, 128)
        r = lambda *s: U.dev(rng.standard_normal(s).astype(np.float16))  # noqa: E731
        z = lambda *s: torch.zeros(s, dtype=torch.float16, device="cuda")  # noqa: E731
        self.fwd, self.bwd = pk.FcPlan(ctx, b, i, n, two_step=True), pk.FcBackwardPlan(ctx, b, i, n)
        self.x, self.target, self.w0 = r(b, i), r(b, n), r(i, n)
        self.w, self.bias, self.y, self.grad, self.gx, self.gw, self.gb = z(i, n), z(n), z(b, n), z(b, n), z(b, i), z(i, n), z(n)
        self.state = [z(i, n), z(i, n), z(n), z(n)]
        torch.cuda.synchronize()
        self.fwd.set_weights(self.w0, self.bias)
        ctx.sync()

    def run(self):
        pk, (_, i, n) = self.pk, self.shape
        self.ctx.call("aig_memcpy", pk.ptr(self.w), pk.ptr(self.w0), 2 * i * n)
        self.fwd.forward(self.x, self.y)
        self.ctx.call("aig_loss_gradient", pk.ptr(self.grad), pk.ptr(self.y), pk.ptr(self.target), self.y.numel())
        self.bwd.backward(self.x, self.grad, self.w, self.gw, self.gb, self.gx)
        mw, vw, mb, vb = self.state
        self.ctx.call("aig_fc_adamw_update", self.fwd.handle, i, n, *(pk.ptr(t) for t in (self.w, self.gw, mw, vw, self.bias, self.gb, mb, vb)), 1e-4, 1, 1e-6)

    def close(self):
        self.fwd.close()
        self.bwd.close()


def _fc_step(U, ctx):
    s = _FcStep(U, ctx)
    return s, s.run, lambda: np.concatenate([U.host(t).ravel() for t in (s.y, s.gx, s.gw, s.w)])


MAKE = {
    "frames in one launch": lambda U, c: _encoder(U, c, 2, 48, 80, (32, 64, 128)),
    "frames layer by layer": lambda U, c: _encoder(U, c, 300, 32, 64, (32, 64)),
    "clips": _clips,
    "sequences": _sequences,
    "fc training step": _fc_step,
}


@gpu
@pytest.mark.parametrize("what", list(MAKE))
def test_switch_reaches_every_launch(env, monkeypatch, what):
    U = env
    edges, results = {}, {}
    U.ctx()
    for off in ("0", "1"):
        monkeypatch.setenv("AIG_NO_PDL", off)
        ctx = U.pkg().Context(0)
        thing, run, result = MAKE[what](U, ctx)
        run()
        ctx.sync()
        results[off] = result()
        ctx.graph_begin()
        run()
        g = ctx.graph_end()
        edges[off] = _programmatic_edges(g)
        U.pkg().lib().aig_graph_destroy(g)
        thing.close()
        ctx.close()
    assert edges["0"] > 0 and edges["1"] == 0, edges
    assert np.array_equal(results["0"], results["1"])
