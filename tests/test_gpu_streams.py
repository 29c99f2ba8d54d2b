"""GPU: a context's scratch serves one stream at a time, and the library enforces it; what may be
captured and replayed beside other work does not use it.

The batched products stage their activations in the context's scratch; two calls issued back
to back on two different streams would otherwise overlap on the device and the second staging
kernel would overwrite what the first product still reads.  The library orders a call behind
the previous scratch user with an event when the stream changes: results must be bit-identical
to the same calls on one stream."""
import numpy as np
import pytest
import torch

from hesper_b200 import BitLinear, Context, GemmaModel, LinearLayer, formats, tp
from tp_common import SMALL_GEMMA

pytestmark = pytest.mark.gpu


def test_batched_calls_on_two_streams_do_not_share_scratch_in_time(ctx):
    rng = np.random.default_rng(9)
    K, N, M = 2560, 4096, 64
    blocks = formats.random_kquant(rng, 12, N, K)
    layer = LinearLayer.create_from_bytes(ctx, blocks, 12, K, N)
    packed = formats.i2s_pack(formats.random_ternary(rng, N, K))
    bl = BitLinear.create_from_bytes(ctx, packed, 0.05, K, N)
    xs = [torch.randn(M, K, device="cuda") for _ in range(6)]
    torch.cuda.synchronize()
    ref_q = [layer.forward(x).clone() for x in xs]
    ref_t = [bl.forward(x).clone() for x in xs]
    torch.cuda.synchronize()
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(5):
        outs_q, outs_t = [], []
        for i, x in enumerate(xs):
            st = sa if i % 2 == 0 else sb
            outs_q.append(layer.forward(x, stream=st))
            outs_t.append(bl.forward(x, stream=sb if i % 2 == 0 else sa))
        sa.synchronize()
        sb.synchronize()
        for i in range(len(xs)):
            assert torch.equal(outs_q[i], ref_q[i]), f"Q4_K call {i}"
            assert torch.equal(outs_t[i], ref_t[i]), f"ternary call {i}"
    ctx.check()


@pytest.mark.parametrize("fmt,M", [(12, 7), (8, 2), (8, 15)])
def test_captured_calls_of_a_few_tokens_share_nothing(ctx, monkeypatch, fmt, M):
    """2 to 15 tokens in a stream capture use no memory of the context: two branches of one graph,
    and its replays beside calls on another stream, do not disturb each other.  That they run on the
    streaming kernel shows in the bits, which are those of a context kept on it."""
    rng = np.random.default_rng(M)
    K, N = 2560, 4096
    blocks = [formats.random_kquant(rng, fmt, N, K) for _ in range(2)]
    layers = [LinearLayer.create_from_bytes(ctx, b, fmt, K, N) for b in blocks]
    x = torch.randn(M, K, device="cuda")
    eager = layers[0].forward(x)
    monkeypatch.setenv("HB200_NO_MMA", "1")
    plain = Context(0)
    monkeypatch.delenv("HB200_NO_MMA")
    want = [LinearLayer.create_from_bytes(plain, b, fmt, K, N).forward(x) for b in blocks]
    torch.cuda.synchronize()
    ys = [torch.empty(M, N, device="cuda") for _ in range(2)]
    g, side, other = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.graph(g):
        main = torch.cuda.current_stream()
        side.wait_stream(main)
        layers[1].forward(x, out=ys[1], stream=side)
        layers[0].forward(x, out=ys[0])
        main.wait_stream(side)
    for _ in range(20):
        for y in ys:
            y.zero_()
        beside = [layers[0].forward(x, stream=other) for _ in range(4)]
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(y, w) for y, w in zip(ys, want))
        assert all(torch.equal(b, eager) for b in beside)
    ctx.check()
    plain.close()


def test_decode_graph_of_a_few_sequences_beside_another_stream(ctx):
    """The engine's graph replays on memory of the engine's own: tokens and products are the same
    with calls of 7 tokens queued on another stream of the same context."""
    w = tp.random_gemma_weights(SMALL_GEMMA, seed=5)
    p = tp.plan(SMALL_GEMMA, 0, 1)
    model = GemmaModel(ctx, SMALL_GEMMA, tp.shard_weights(SMALL_GEMMA, w, p), p, None, batch=4, max_new_tokens=40)
    prompt = np.arange(12, dtype=np.int32).reshape(4, 3)
    model.generate(prompt, 2)
    model.set_position(3)
    want, _, _ = model.generate(None, 30)
    rng = np.random.default_rng(0)
    layer = LinearLayer.create_from_bytes(ctx, formats.random_kquant(rng, 12, 4096, 2560), 12, 2560, 4096)
    x = torch.randn(7, 2560, device="cuda")
    ref = layer.forward(x)
    other = torch.cuda.Stream()
    for _ in range(5):
        model.generate(prompt, 2)
        model.set_position(3)
        torch.cuda.synchronize()
        outs = [layer.forward(x, stream=other) for _ in range(400)]
        got, _, _ = model.generate(None, 30)
        torch.cuda.synchronize()
        assert np.array_equal(got, want)
        assert all(torch.equal(o, ref) for o in outs)
    ctx.check()
    model.close()


@pytest.mark.parametrize("gate_up", [False, True])
def test_captured_rows_too_long_for_the_streaming_kernel(ctx, gate_up):
    """Rows that only the kernel for a few tokens takes are captured on it, with the context's scratch
    as the batched products are."""
    rng = np.random.default_rng(3)
    K, N, M = 16384, 40, 5
    a, b = (LinearLayer.create_from_bytes(ctx, formats.random_kquant(rng, 8, N, K), 8, K, N) for _ in "ab")
    x = torch.randn(M, K, device="cuda")

    def call():
        return LinearLayer.forward_fused_gate_up(a, b, x) if gate_up else a.forward(x)
    want, g = call(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = call()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    ctx.check()
