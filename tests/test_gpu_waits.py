"""GPU: a kernel launched early waits for its predecessor without a deadline.

With programmatic dependent launch the batched products are resident, their weights prefetched,
while an earlier kernel of the stream still runs.  Their waits on mbarriers are bounded; none that
depends on that kernel's results may start before it has ended.  The predecessor here is the
one-warp bit-reproducible attention kernel over 2 M positions: about a second on one warp."""
import numpy as np
import pytest
import torch

from hesper_b200 import BitLinear, LinearLayer, _lib, execute_flash_attention_v11, formats

pytestmark = pytest.mark.gpu


def _kquant(ctx, rng, fmt, M):
    K, N = 2560, 1500
    layer = LinearLayer.create_from_bytes(ctx, formats.random_kquant(rng, fmt, N, K), fmt, K, N)
    x = torch.randn(M, K, device="cuda")
    return lambda: layer.forward(x)


def _ternary(ctx, rng, M):
    K, N = 6912, 1500
    layer = BitLinear.create_from_bytes(ctx, formats.i2s_pack(formats.random_ternary(rng, N, K)), 0.05, K, N)
    x = torch.randn(M, K, device="cuda")
    return lambda: layer.forward(x)


def _lmhead(ctx, M):
    K, V = 2560, 148 * 128 * 2
    table = torch.randn(V, K, device="cuda").bfloat16()
    x, logits = torch.randn(M, K, device="cuda"), torch.empty(M, V, device="cuda")
    tok = torch.empty(M, dtype=torch.int32, device="cuda")
    lib = _lib.load()
    keys = torch.zeros(lib.hb200_lmhead_scratch_bytes(M), dtype=torch.uint8, device="cuda")

    def call():
        _lib.check(lib.hb200_lmhead_argmax(ctx.handle, table.data_ptr(), 0, V, K, x.data_ptr(), M, None, 0.0,
                                           logits.data_ptr(), tok.data_ptr(), keys.data_ptr(), None, None, 0,
                                           torch.cuda.current_stream().cuda_stream))
        return logits.clone()
    return call


@pytest.mark.parametrize("what", ["q4k 5", "q4k 16", "q4k 100", "q4k 200", "q8_0 16", "ternary 16", "ternary 128",
                                  "lmhead 20"])
def test_products_outwait_a_long_predecessor(ctx, what):
    kind, M = what.split()
    M, rng = int(M), np.random.default_rng(len(what))
    call = {"q4k": lambda: _kquant(ctx, rng, 12, M), "q8_0": lambda: _kquant(ctx, rng, 8, M),
            "ternary": lambda: _ternary(ctx, rng, M), "lmhead": lambda: _lmhead(ctx, M)}[kind]()
    want = call()
    L, D = 1 << 21, 64
    q = torch.randn(1, 1, D, device="cuda")
    kv = torch.randn(1, 1, L, D, device="cuda", dtype=torch.float16)
    sl = torch.tensor([L], dtype=torch.int32, device="cuda")
    ctx.check()
    s, e = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    try:
        ctx.set_attn_mode(ctx.ATTN_EXACT)
        s.record()
        execute_flash_attention_v11(ctx, q, kv, kv, sl, num_heads=1, num_kv_heads=1, head_dim=D, max_seq_len=L,
                                    scale=0.1)
        got = call()
        e.record()
        ctx.check()
    finally:
        ctx.set_attn_mode(ctx.ATTN_FAST)
    assert torch.equal(got, want)
    assert s.elapsed_time(e) > 300  # ms: the predecessor was long enough to matter
