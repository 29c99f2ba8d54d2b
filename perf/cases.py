"""The work that a program built on this framework has it do, as cases that can be timed.

Every case goes through the public entry points: the layer API (`hesper_b200.layers`), the C ABI
where the layer API has no wrapper (LM head, decode loop with the caller's own sampler) and the
Gemma-shaped decode engine.  Sizes are those of the two model shapes the repository is built
around (`BitNetShape`, `GemmaShape`) and of its benchmark; `draw` spreads them over the ranges
that the entry points take.

Operator cases hold a stack of distinct layers and run each once per pass, as the layers of a
model follow one another, so that weights and caches come from device memory and not from L2.

The full-depth BitNet decode loop is covered by its operators and not as a whole: a randomly
initialised model re-quantises its activations to int8 in every block, so that two correct
attention kernels that differ in the last bit end in different tokens, and there is no tolerance
to compare them with.  The Q4_K model has no such step and is run whole.
"""
import functools
import math
import weakref

import torch

import hesper_b200 as hb
from hesper_b200 import _lib
from hesper_b200 import layers as hl
from hesper_b200 import tp as htp

Q8_0, Q4_K = 8, 12


def listed():
    return [
        # One token through the ternary layers of BitNet-2B blocks (q/k/v, o_proj, gate/up,
        # down): batch-1 decode, the smallest calls there are.
        dict(name="ternary_decode_m1", kind="ternary", tokens=1, hidden=2560, kv=640, ffn=6912, depth=6),
        # The same blocks on a prompt chunk.
        dict(name="ternary_prompt_m256", kind="ternary", tokens=256, hidden=2560, kv=640, ffn=6912, depth=6),
        # One token, Q4_K, the benchmark's headline matrix.
        dict(name="q4k_m1", kind="kquant", op="linear", fmt=Q4_K, tokens=1, K=2560, N=10240, depth=8),
        # A handful of sequences decoded together on Q8_0 weights.
        dict(name="q8_0_m7", kind="kquant", op="linear", fmt=Q8_0, tokens=7, K=2560, N=10240, depth=4),
        # Gated FFN input (norm, gate, up, GeGLU) for a serving batch.
        dict(name="q4k_geglu_m64", kind="kquant", op="gate_up", fmt=Q4_K, tokens=64, K=2560, N=10240, depth=4),
        # Decode attention of one sequence over a medium cache: latency.
        dict(name="attn_b1_l4096", kind="attn", seqs=1, new=0, heads=8, kv_heads=2, head_dim=256, slots=4096, window=0, depth=8),
        # Decode attention of a full serving batch with ragged lengths: bandwidth.
        dict(name="attn_b64_l8192", kind="attn", seqs=64, new=0, heads=8, kv_heads=2, head_dim=256, slots=8192, window=0, depth=1),
        # Prompt chunk at the end of a long context.
        dict(name="attn_prompt_t256", kind="attn", seqs=1, new=256, heads=8, kv_heads=2, head_dim=256, slots=8192, window=0, depth=4),
        # LM head with final norm and argmax for a serving batch.
        dict(name="lmhead_m32", kind="lmhead", tokens=32, vocab=128256, K=2560, depth=1),
        # A short interactive exchange: greedy generation, one sequence.
        dict(name="gemma_generate_b1", kind="generate", prompt=12, steps=24),
        # 32 sequences served together: short prompts, then decode steps whose tokens the caller
        # picks (its own sampler reads the logits).
        dict(name="gemma_serve_b32", kind="serve", seqs=32, prompt=16, steps=8),
        # A long prompt of one sequence up to its first token's logits.
        dict(name="gemma_prompt_2048", kind="serve", seqs=1, prompt=2048, steps=0),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _depth(weight_bytes):
    """Layers in a stack: enough for about 96 MB of weights or caches, at most 12."""
    return max(1, min(12, int(96e6 // max(1, weight_bytes)) + 1))


def draw(rng):
    kind = rng.choice(["ternary", "ternary", "kquant", "kquant", "kquant", "attn", "attn", "prompt_attn",
                       "lmhead", "generate", "serve"])
    if kind == "ternary":
        hidden, ffn = 128 * rng.randint(8, 32), 128 * rng.randint(16, 72)
        kv = 64 * rng.randint(2, hidden // 128)
        per = (hidden * (2 * hidden + 2 * kv) + 3 * hidden * ffn) // 4
        return dict(kind=kind, tokens=_log_int(rng, 1, 400), hidden=hidden, kv=kv, ffn=ffn, depth=_depth(per))
    if kind == "kquant":
        op, fmt = rng.choice(["linear", "linear", "qkv", "gate_up"]), rng.choice([Q4_K, Q4_K, Q8_0])
        K, N = 256 * _log_int(rng, 4, 40), _log_int(rng, 500, 14000)
        per = N * K * (144 / 256 if fmt == Q4_K else 34 / 32) * (2 if op == "gate_up" else 1)
        return dict(kind=kind, op=op, fmt=fmt, tokens=_log_int(rng, 1, 400), K=K, N=N, depth=_depth(per))
    if kind in ("attn", "prompt_attn"):
        D = rng.choice([64, 128, 256])
        G = rng.choice([1, 2, 4, 8])
        kv_heads = rng.randint(1, 5)
        new = 0 if kind == "attn" else _log_int(rng, 8, 512)
        seqs = _log_int(rng, 1, 64) if kind == "attn" else rng.randint(1, 4)
        slots = max(_log_int(rng, 100, 16384), 2 * new)
        # at most the listed batch's cache
        slots = max(2 * new, 100, min(slots, int(1.0e9 / (seqs * kv_heads * 4 * D))))
        if new:  # at most four times the listed chunk's products
            slots = max(2 * new, min(slots, int(6.8e10 / (4.0 * new * seqs * kv_heads * G * D))))
        window = rng.choice([0, 0, 0, 512])
        return dict(kind="attn", seqs=seqs, new=new, heads=G * kv_heads, kv_heads=kv_heads, head_dim=D,
                    slots=slots, window=window, depth=_depth(4 * seqs * kv_heads * slots * D))
    if kind == "lmhead":
        V, K = _log_int(rng, 16000, 262144), 64 * rng.randint(16, 48)
        return dict(kind=kind, tokens=_log_int(rng, 1, 64), vocab=V, K=K, depth=1)
    if kind == "generate":
        return dict(kind=kind, prompt=rng.randint(2, 15), steps=rng.randint(8, 21))
    seqs = _log_int(rng, 2, 64)
    return dict(kind="serve", seqs=seqs, prompt=_log_int(rng, 4, max(8, 512 // seqs)), steps=rng.randint(1, 3))


# ---- inputs -------------------------------------------------------------------------------------


@functools.lru_cache(maxsize=1)
def _context():
    """A program has one context per GPU."""
    return hb.Context(torch.cuda.current_device())


def _ternary_layer(ctx, gen, K, N):
    """i2_s bytes with P(-1, 0, +1) = 1/4, 1/2, 1/4 (code = value + 1) and one scale."""
    u = torch.randint(0, 4, (4, N * K // 4), device="cuda", generator=gen, dtype=torch.uint8)
    c = (u + 1) // 2
    packed = (c[0] << 6) | (c[1] << 4) | (c[2] << 2) | c[3]
    scale = torch.empty(1, device="cuda").uniform_(0.01, 0.1, generator=gen)
    return hl.BitLinear(ctx, packed, scale, K, N)


def _kquant_layer(ctx, gen, fmt, K, N):
    if fmt == Q4_K:
        return hl.LinearLayer(ctx, htp.random_q4k_device(N * (K // 256), gen), hl.QuantFormat.Q4_K, K, N)
    nb = N * (K // 32)
    blocks = torch.empty((nb, 34), dtype=torch.uint8, device="cuda")
    d = torch.empty(nb, device="cuda").uniform_(1e-3, 1e-2, generator=gen).half()
    blocks[:, :2] = d.view(torch.uint8).reshape(nb, 2)
    blocks[:, 2:] = torch.randint(-127, 128, (nb, 32), device="cuda", generator=gen, dtype=torch.int8).view(torch.uint8)
    return hl.LinearLayer(ctx, blocks.reshape(-1), hl.QuantFormat.Q8_0, K, N)


def _randn(gen, *shape):
    return torch.randn(*shape, device="cuda", generator=gen)


def _gain(gen, n):
    return 1.0 + 0.05 * _randn(gen, n)


def _prepare_ternary(c, ctx, gen):
    H, F, M = c["hidden"], c["ffn"], c["tokens"]
    blocks = []
    for _ in range(c["depth"]):
        blocks.append(dict(
            qkv=[_ternary_layer(ctx, gen, H, n) for n in (H, c["kv"], c["kv"])],
            o=_ternary_layer(ctx, gen, H, H), gate=_ternary_layer(ctx, gen, H, F),
            up=_ternary_layer(ctx, gen, H, F), down=_ternary_layer(ctx, gen, F, H),
            norm=_gain(gen, H), sub_norm=_gain(gen, H), ffn_norm=_gain(gen, H), ffn_sub_norm=_gain(gen, F),
            att=_randn(gen, M, H)))
    return dict(blocks=blocks, x=_randn(gen, M, H))


def _run_ternary(s):
    """Blocks one after another; attention itself is a case of its own, its output is given."""
    x, out = s["x"], []
    for b in s["blocks"]:
        out += hl.BitLinear.forward_multi(b["qkv"], x, rms_gamma=b["norm"])
        h = b["o"].forward_fused_rmsnorm_residual(b["att"], b["sub_norm"], x)
        a = hl.BitLinear.forward_fused_gate_up_relu_sqr_mul(b["gate"], b["up"], h, rms_gamma=b["ffn_norm"])
        x = b["down"].forward_fused_rmsnorm_residual(a, b["ffn_sub_norm"], h)
    return out + [x]


def _prepare_kquant(c, ctx, gen):
    K, N, fmt = c["K"], c["N"], c["fmt"]
    parts = {"linear": [N], "gate_up": [N, N], "qkv": [N, max(1, N // 4), max(1, N // 4)]}[c["op"]]
    stack = [[_kquant_layer(ctx, gen, fmt, K, n) for n in parts] for _ in range(c["depth"])]
    return dict(op=c["op"], stack=stack, x=_randn(gen, c["tokens"], K), norms=[_gain(gen, K) for _ in stack])


def _run_kquant(s):
    if s["op"] == "linear":
        return [layer[0].forward(s["x"]) for layer in s["stack"]]
    if s["op"] == "gate_up":
        return [hl.LinearLayer.forward_fused_gate_up(layer[0], layer[1], s["x"], rms_gamma=g)
                for layer, g in zip(s["stack"], s["norms"])]
    return [hl.LinearLayer.forward_multi(layer, s["x"], rms_gamma=g) for layer, g in zip(s["stack"], s["norms"])]


def _prepare_attn(c, ctx, gen):
    B, T, L, D = c["seqs"], c["new"], c["slots"], c["head_dim"]
    kv = (B, c["kv_heads"], L, D)
    caches = [tuple(torch.empty(kv, dtype=torch.float16, device="cuda").normal_(generator=gen) for _ in "kv")
              for _ in range(c["depth"])]
    # one sequence fills its cache; of several each has its own length
    low = L if B == 1 else max(T, L // 2, 1)
    lens = torch.randint(low, L + 1, (B,), device="cuda", generator=gen, dtype=torch.int32)
    q = _randn(gen, B, T, c["heads"], D) if T else _randn(gen, B, c["heads"], D)
    args = dict(num_heads=c["heads"], num_kv_heads=c["kv_heads"], head_dim=D, max_seq_len=L,
                scale=D ** -0.5, window=c["window"])
    if not T:  # decode loops keep the partials' workspace
        args["workspace"] = hl.flash_attention_workspace(ctx, B, c["heads"], c["kv_heads"], D, L)
    return dict(ctx=ctx, caches=caches, lens=lens, q=q, args=args,
                call=hl.flash_attention_prefill if T else hl.execute_flash_attention_v11)


def _run_attn(s):
    return [s["call"](s["ctx"], s["q"], k, v, s["lens"], **s["args"]) for k, v in s["caches"]]


def _prepare_lmhead(c, ctx, gen):
    M, V, K = c["tokens"], c["vocab"], c["K"]
    table = (0.02 * _randn(gen, V, K)).to(torch.bfloat16)
    return dict(ctx=ctx, table=table, x=_randn(gen, M, K), gamma=_gain(gen, K), M=M, V=V, K=K,
                logits=torch.empty(M, V, device="cuda"), tok=torch.empty(M, dtype=torch.int32, device="cuda"),
                keys=torch.zeros(_lib.load().hb200_lmhead_scratch_bytes(M), dtype=torch.uint8, device="cuda"))


def _run_lmhead(s):
    _lib.check(_lib.load().hb200_lmhead_argmax(
        s["ctx"].handle, s["table"].data_ptr(), 0, s["V"], s["K"], s["x"].data_ptr(), s["M"],
        s["gamma"].data_ptr(), 1e-5, s["logits"].data_ptr(), s["tok"].data_ptr(), s["keys"].data_ptr(),
        None, None, 0, torch.cuda.current_stream().cuda_stream))
    return s["logits"], s["tok"]


class _Logits:
    """The engine's own [B][vocab] buffer; a tensor over it keeps the model alive."""

    def __init__(self, model, batch, vocab):
        self.model = model
        self.__cuda_array_interface__ = {
            "shape": (batch, vocab), "typestr": "<f4", "version": 2,
            "data": (int(_lib.load().hb200_gemma_local_logits(model._h)), False)}


def _prepare_gemma(c, ctx, gen, seed):
    """The Gemma-4-E4B-shaped model of the repository with random Q4_K weights."""
    shape = htp.GemmaShape()
    plan = htp.plan(shape, 0, 1)
    B, P, S = c.get("seqs", 1), c["prompt"], c["steps"]
    model = htp.GemmaModel(ctx, shape, htp.random_gemma_shard_device(shape, plan, seed=seed), plan,
                           batch=B, max_new_tokens=max(1, S + 2))
    weakref.finalize(model, _lib.load().hb200_gemma_destroy, model._h)
    ids = torch.randint(0, shape.vocab, (B, P + S), device="cuda", generator=gen, dtype=torch.int32)
    s = dict(ctx=ctx, model=model, steps=S)
    if c["kind"] == "generate":
        return dict(s, prompt=ids[:, :P].cpu().numpy())
    T = model.chunk
    s["chunks"] = [ids[:, i:min(i + T, P)].contiguous() for i in range(0, P, T)]
    s["next"] = [ids[:, P + j].contiguous() for j in range(S)]

    s["logits"] = torch.as_tensor(_Logits(model, B, shape.vocab), device="cuda")
    return s


def _run_generate(s):
    return s["model"].generate(s["prompt"], s["steps"])[0]


def _run_serve(s):
    """Prompt in passes, then decode steps on tokens the caller chose; the last logits."""
    lib, h = _lib.load(), s["model"]._h
    st = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.hb200_gemma_reset(h, st))
    for ids in s["chunks"]:
        _lib.check(lib.hb200_gemma_prefill(h, ids.data_ptr(), ids.shape[1], int(ids is s["chunks"][-1]), st))
    for ids in s["next"]:
        _lib.check(lib.hb200_gemma_step(h, ids.data_ptr(), st))
    return s["logits"]


def prepare(case, seed):
    ctx = _context()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind in ("generate", "serve"):
        return dict(_prepare_gemma(case, ctx, gen, seed), kind=kind)
    return dict({"ternary": _prepare_ternary, "kquant": _prepare_kquant, "attn": _prepare_attn,
                 "lmhead": _prepare_lmhead}[kind](case, ctx, gen), kind=kind)


def run(state):
    return {"ternary": _run_ternary, "kquant": _run_kquant, "attn": _run_attn, "lmhead": _run_lmhead,
            "generate": _run_generate, "serve": _run_serve}[state["kind"]](state)


# ---- what a pass cannot do without -----------------------------------------------------------------


def _attn_work(c):
    """Expected lengths; every cached position that a query sees is read once per KV head."""
    B, T, L, D, W = c["seqs"], c["new"], c["slots"], c["head_dim"], c["window"]
    n = L if B == 1 else 0.5 * (L + max(T, L // 2, 1))
    t = max(1, T)
    seen = min(n, W + t - 1) if W else n              # positions some query of the chunk sees
    pairs = t * (min(n, W) if W else n - 0.5 * (t - 1))  # (query, position) pairs
    kv = 2 * 2 * B * c["kv_heads"] * seen * D
    io = B * t * c["heads"] * D * 8
    return dict(bytes=kv + io, flops=4.0 * B * c["heads"] * pairs * D)


def work(case):
    c, kind = case, case["kind"]
    if kind == "ternary":
        H, F, M, KV, n = c["hidden"], c["ffn"], c["tokens"], c["kv"], c["depth"]
        weights = H * (H + 2 * KV) + H * H + 3 * H * F
        acts = 4 * M * (H + H + 2 * KV + H)           # hidden state in; q, k, v out; attention output in
        return dict(bytes=n * (weights / 4 + acts) + 4 * M * H, flops=2.0 * n * M * weights)
    if kind == "kquant":
        K, N, M, n = c["K"], c["N"], c["tokens"], c["depth"]
        rows = {"linear": N, "gate_up": 2 * N, "qkv": N + 2 * max(1, N // 4)}[c["op"]]
        out = N if c["op"] == "gate_up" else rows
        per = 144 / 256 if c["fmt"] == Q4_K else 34 / 32
        return dict(bytes=n * (rows * K * per + 4 * M * out) + 4 * M * K, flops=2.0 * n * M * rows * K)
    if kind == "attn":
        w = _attn_work(c)
        return dict(bytes=c["depth"] * w["bytes"], flops=c["depth"] * w["flops"])
    if kind == "lmhead":
        M, V, K = c["tokens"], c["vocab"], c["K"]
        return dict(bytes=2 * V * K + 4 * M * (K + V), flops=2.0 * M * V * K)
    s = htp.GemmaShape()
    B, P, S = c.get("seqs", 1), c["prompt"], c["steps"]
    q, kv = s.n_heads * s.head_dim, s.n_kv_heads * s.head_dim
    block = s.hidden * (2 * q + 2 * kv + 3 * s.ffn) * s.n_layers
    head = s.hidden * s.vocab
    heads = S if kind == "generate" else S + 1        # passes that end in logits
    decode = S - 1 if kind == "generate" else S
    passes = 1 + decode                               # the whole prompt could be one pass
    L = P + decode
    kv_bytes = 4 * B * kv * s.n_layers * (P + sum(P + 1 + j for j in range(decode)))
    attn = 4.0 * B * q * s.n_layers * L * (L + 1) / 2
    return dict(bytes=0.5625 * (passes * block + heads * head) + kv_bytes + 4 * heads * B * s.vocab,
                flops=2.0 * B * (block * L + head * heads) + attn)


def tolerance(case):
    kind = case["kind"]
    if kind == "ternary":
        return {"rel": 1e-6, "max": 1e-4}   # integer products; f32 epilogues
    if kind == "kquant":                    # 16-bit block-quantised activations; f16 operands from 16 tokens on
        return {"rel": 1e-4} if case["tokens"] < 16 else {"rel": 1e-3}
    if kind == "attn":
        return {"rel": 1e-3}                # f16 softmax weights and query
    if kind == "lmhead":
        return {"rel": 2e-5, "differ": 0.01}  # 16-bit table, activations in two terms
    if kind == "generate":
        return {"rel": 0.0, "differ": 0.01}   # greedy tokens
    return {"rel": 3e-3}                    # f16 products and attention through 42 layers
