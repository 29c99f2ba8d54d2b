"""GPU parity: Q4_K / Q8_0 dequant-fused matvec through the C ABI vs the f64 oracle.
Bar (stated by the task for k-quant outputs): relative error <= 1e-3.  Measured as
max |y - ref| / max |ref| and as relative L2; the kernel sits near 1e-5."""
import numpy as np
import pytest
import torch

import hesper_b200 as hb
from hesper_b200 import LinearLayer, QuantFormat, formats
from test_oracle_kquant import reference_q4k_block

pytestmark = pytest.mark.gpu

TOL = 1e-3


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _check(y, ref, tol=TOL):
    y = y.cpu().numpy().astype(np.float64)
    ref = ref.astype(np.float64)
    scale = np.max(np.abs(ref)) + 1e-30
    assert np.max(np.abs(y - ref)) / scale <= tol
    assert np.linalg.norm(y - ref) / (np.linalg.norm(ref) + 1e-30) <= tol
    return np.max(np.abs(y - ref)) / scale


@pytest.mark.parametrize("fmt", [12, 8])
@pytest.mark.parametrize("K,N", [(2560, 10240), (2560, 2048), (2560, 512), (2048, 2560),
                                 (10240, 2560), (256, 1), (512, 7), (768, 33), (4096, 1000)])
def test_matvec_shapes(ctx, oracle, fmt, K, N):
    rng = np.random.default_rng(K + 3 * N + fmt)
    blocks = formats.random_kquant(rng, fmt, N, K)
    x = rng.standard_normal((1, K)).astype(np.float32)
    ref = oracle.kquant_matvec(fmt, blocks, K, N, x)
    layer = LinearLayer.create_from_bytes(ctx, blocks, fmt, K, N)
    y = layer.forward(_dev(x))
    ctx.check()
    err = _check(y, ref)
    assert err < 2e-4  # the kernel's own design point: 16-bit block-scaled activations


@pytest.mark.parametrize("fmt", [12, 8])
@pytest.mark.parametrize("M", [2, 17])
def test_streaming_kernel_several_tokens(oracle, monkeypatch, fmt, M):
    """The streaming kernel sends every token around its ring of weight tiles again.  18 and 35
    tiles per CTA on 12 warps: some warps hold a tile more than others, so the second token starts
    at different ring positions."""
    monkeypatch.setenv("HB200_NO_MMA", "1")
    K, N = 2560, 10240
    rng = np.random.default_rng(M + fmt)
    blocks = formats.random_kquant(rng, fmt, N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    c = hb.Context(0)
    y = LinearLayer.create_from_bytes(c, blocks, fmt, K, N).forward(_dev(x))
    c.check()
    c.close()
    rows = [0, 1, M - 1]
    assert _check(y[rows], oracle.kquant_matvec(fmt, blocks, K, N, x[rows])) < 2e-4


def test_reference_block_fixture(ctx, oracle):
    blk = reference_q4k_block(42)
    x = np.sin(0.1 * np.arange(256)).astype(np.float32)
    ref = oracle.q4k_matvec(blk, 256, 1, x)
    y = LinearLayer.create_from_bytes(ctx, blk, 12, 256, 1).forward(_dev(x[None, :]))
    _check(y, ref)


@pytest.mark.parametrize("fmt", [12, 8])
@pytest.mark.parametrize("M", [1, 2, 5])
def test_residual_rmsnorm_batch(ctx, oracle, fmt, M):
    K, N = 2560, 300
    rng = np.random.default_rng(17 * M + fmt)
    blocks = formats.random_kquant(rng, fmt, N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    gamma = (1.0 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    res = rng.standard_normal((M, N)).astype(np.float32)
    layer = LinearLayer.create_from_bytes(ctx, blocks, fmt, K, N)
    ref = oracle.kquant_matvec(fmt, blocks, K, N, x, residual=res)
    _check(layer.forward(_dev(x), residual=_dev(res)), ref)
    xn = np.stack([oracle.rmsnorm_f64(x[m], gamma, 1e-6) for m in range(M)]).astype(np.float32)
    ref = oracle.kquant_matvec(fmt, blocks, K, N, xn)
    _check(layer.forward(_dev(x), rms_gamma=_dev(gamma), eps=1e-6), ref)
    ctx.check()


@pytest.mark.parametrize("fmt", [12, 8])
@pytest.mark.parametrize("K,N,M", [(2560, 10240, 1), (256, 3, 1), (2560, 130, 2)])
def test_gate_up_gelu(ctx, oracle, fmt, K, N, M):
    rng = np.random.default_rng(K + N + M + fmt)
    bg = formats.random_kquant(rng, fmt, N, K)
    bu = formats.random_kquant(rng, fmt, N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    ref = oracle.kquant_gateup_gelu(bg, bu, fmt, K, N, x)
    g = LinearLayer.create_from_bytes(ctx, bg, fmt, K, N)
    u = LinearLayer.create_from_bytes(ctx, bu, fmt, K, N)
    y = LinearLayer.forward_fused_gate_up(g, u, _dev(x))
    ctx.check()
    _check(y, ref)


@pytest.mark.parametrize("fmt", [12, 8])
@pytest.mark.parametrize("K,Ns,M,gate_up", [
    (256, [1], 3, False),            # one super-block, one row: most warps idle
    (768, [5, 640], 8, False),       # rows of two tensors on disjoint CTAs, all 8 columns of a tile
    (2560, [2048, 512, 130], 9, False),  # second column tile with one token
    (512, [148 * 128 + 37], 15, False),  # two passes per CTA, the second one ragged
    (1024, [148 * 64 + 11], 3, True),    # gate/up, two passes
    (2560, [333], 12, True), (2560, [2600], 2, False),
    # two tokens on either side of the rule: Q8_0 10 M weights; Q4_K rows >= 4 K, 16 M weights
    (1024, [9765], 2, False), (1024, [9766], 2, False), (768, [3071], 2, False), (768, [3072], 2, False),
    (3840, [4166], 2, False), (3840, [4167], 2, False), (1024, [2047], 2, True), (1024, [2048], 2, True),
    # the ring of weights wraps (tests/test_kquant_few_tokens_plan.py): one tile per CTA and fewer
    # stages than warps; unequal tensors; several laps; two passes
    (4096, [2304], 15, False), (9216, [2304], 9, False), (4096, [1152], 12, True),
    (4096, [1536, 384, 384], 12, False), (4096, [11000, 16], 3, False),
    (10240, [2560], 7, False), (10240, [2560], 15, False),
    (4096, [148 * 128 + 37], 3, False), (4096, [148 * 64 + 11], 12, True)])
def test_few_tokens(ctx, oracle, fmt, K, Ns, M, gate_up):
    """2 to 15 tokens: 16-bit block-quantised activations, exact integer products.  An activation
    is off by at most 2^-16 of its block's largest: 2e-4 of max|y| as for one token."""
    rng = np.random.default_rng(K + sum(Ns) + M + fmt)
    x = rng.standard_normal((M, K)).astype(np.float32)
    gamma = (1.0 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    xn = np.stack([oracle.rmsnorm_f64(x[m], gamma, 1e-6) for m in range(M)]).astype(np.float32)
    if gate_up:
        bg, bu = (formats.random_kquant(rng, fmt, Ns[0], K) for _ in range(2))
        g, u = (LinearLayer.create_from_bytes(ctx, b, fmt, K, Ns[0]) for b in (bg, bu))
        y = LinearLayer.forward_fused_gate_up(g, u, _dev(x), rms_gamma=_dev(gamma), eps=1e-6)
        ctx.check()
        assert _check(y, oracle.kquant_gateup_gelu(bg, bu, fmt, K, Ns[0], xn)) < 2e-4
        return
    blocks = [formats.random_kquant(rng, fmt, n, K) for n in Ns]
    layers = [LinearLayer.create_from_bytes(ctx, b, fmt, K, n) for b, n in zip(blocks, Ns)]
    res = rng.standard_normal((M, Ns[0])).astype(np.float32)
    y = layers[0].forward(_dev(x), residual=_dev(res))
    assert _check(y, oracle.kquant_matvec(fmt, blocks[0], K, Ns[0], x, residual=res)) < 2e-4
    ys = LinearLayer.forward_multi(layers, _dev(x), rms_gamma=_dev(gamma), eps=1e-6)
    ctx.check()
    for b, n, y in zip(blocks, Ns, ys):
        assert _check(y, oracle.kquant_matvec(fmt, b, K, n, xn)) < 2e-4


def test_two_contexts_share_a_kernel_of_different_shared_memory(oracle, monkeypatch):
    """Two contexts of one GPU, the same kernel with much and with little shared memory: neither's call
    takes the other's back."""
    monkeypatch.setenv("HB200_NO_MMA", "1")
    rng = np.random.default_rng(8)
    big, small = hb.Context(0), hb.Context(0)
    wb, ws = formats.random_kquant(rng, 12, 10240, 2560), formats.random_kquant(rng, 12, 8, 256)
    lb, ls = LinearLayer.create_from_bytes(big, wb, 12, 2560, 10240), LinearLayer.create_from_bytes(small, ws, 12, 256, 8)
    x = rng.standard_normal((2, 2560)).astype(np.float32)
    ref = oracle.kquant_matvec(12, wb, 2560, 10240, x)
    _check(lb.forward(_dev(x)), ref)
    ls.forward(torch.zeros(2, 256, device="cuda"))
    _check(lb.forward(_dev(x)), ref)
    for c in (big, small):
        c.check()
        c.close()


@pytest.mark.parametrize("M", [1, 5, 20])
def test_half_a_pre_step_is_refused(ctx, M):
    K, N = 256, 64
    rng = np.random.default_rng(0)
    a, b = (LinearLayer.create_from_bytes(ctx, formats.random_kquant(rng, 12, N, K), 12, K, N) for _ in "ab")
    x, base, gamma = (torch.randn(n, K, device="cuda") for n in (M, M, 1))
    for pre in ((base, None), (None, gamma), (None, None)):
        with pytest.raises(hb.HesperB200Error, match="null"):
            LinearLayer.forward_multi([a, b], x, pre=pre)
        with pytest.raises(hb.HesperB200Error, match="null"):
            LinearLayer.forward_fused_gate_up(a, b, x, pre=pre)
    with pytest.raises(ValueError):
        LinearLayer.forward_fused_gate_up(a, b, x, pre=(base,))
    y, xo = LinearLayer.forward_fused_gate_up(a, b, x, pre=(base, gamma))
    ys, xo2 = LinearLayer.forward_multi([a, b], x, pre=[base, gamma])
    assert torch.equal(xo, xo2) and y.shape == ys[1].shape == (M, N)
    ctx.check()


def test_an_output_that_does_not_fit_is_an_out_of_memory_error(ctx):
    rng = np.random.default_rng(0)
    layer = LinearLayer.create_from_bytes(ctx, formats.random_kquant(rng, 12, 8, 256), 12, 256, 8)
    layer.out_dim = 2 ** 31 - 1  # 35 TB of output for 4096 tokens; nothing is launched
    with pytest.raises(torch.OutOfMemoryError):
        layer.forward(torch.zeros(4096, 256, device="cuda"))


@pytest.mark.parametrize("M", [16, 100, 200])
def test_minima_beyond_f16(ctx, oracle, M):
    """dmin * m far above f16's largest value, next to weights that f16 holds (d * sc * q cancels it):
    every third row has such blocks, from the smallest dmin whose product with 63 is out of range."""
    K, N = 512, 200
    rng = np.random.default_rng(M)
    nb = N * (K // 256)
    d, dmin = np.full(nb, 0.01), np.full(nb, 0.02)
    sc, m = rng.integers(0, 64, (nb, 8)), rng.integers(0, 64, (nb, 8))
    q = rng.integers(0, 16, (nb, 256))
    for i in range(0, nb, 3):
        if i % 2:  # 60 * 1100 * {14, 15} - 63 * 15000 = -21000, 45000
            d[i], dmin[i], sc[i], m[i] = 1100.0, 15000.0, 60, 63
            q[i] = rng.integers(14, 16, 256)
        else:      # 62 * 75 * {13 .. 15} - 63 * 1040: 65520 rounds to infinity in f16
            d[i], dmin[i], sc[i], m[i] = 75.0, 1040.0, 62, 63
            q[i] = rng.integers(13, 16, 256)
    blocks = formats.q4k_build(d, dmin, sc, m, q).reshape(-1)
    x = rng.standard_normal((M, K)).astype(np.float32)
    y = LinearLayer.create_from_bytes(ctx, blocks, 12, K, N).forward(_dev(x))
    ctx.check()
    assert _check(y, oracle.kquant_matvec(12, blocks, K, N, x)) < 1e-3


@pytest.mark.parametrize("fmt", [12, 8])
@pytest.mark.parametrize("M", [16, 64])
def test_longest_rows_of_the_batched_product(ctx, oracle, fmt, M):
    """K = 65280 is the longest row 16 tokens or more take, in both formats; 65536 is refused."""
    K, N = 65280, 70
    rng = np.random.default_rng(fmt + M)
    blocks = formats.random_kquant(rng, fmt, N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    y = LinearLayer.create_from_bytes(ctx, blocks, fmt, K, N).forward(_dev(x))
    ctx.check()
    rows = [0, 9, M - 1]
    assert _check(y[rows], oracle.kquant_matvec(fmt, blocks, K, N, x[rows])) < 1e-3
    long = LinearLayer.create_from_bytes(ctx, formats.random_kquant(rng, fmt, 8, 65536), fmt, 65536, 8)
    with pytest.raises(hb.HesperB200Error):
        long.forward(torch.zeros(M, 65536, device="cuda"))


def test_fused_qkv_multi(ctx, oracle):
    K = 2560
    rng = np.random.default_rng(8)
    shapes = [2048, 512, 512]
    blocks = [formats.random_q4k(rng, n, K) for n in shapes]
    x = rng.standard_normal((1, K)).astype(np.float32)
    gamma = (1.0 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    layers = [LinearLayer.create_from_bytes(ctx, b, 12, K, n) for b, n in zip(blocks, shapes)]
    ys = LinearLayer.forward_multi(layers, _dev(x), rms_gamma=_dev(gamma), eps=1e-6)
    ctx.check()
    xn = oracle.rmsnorm_f64(x[0], gamma, 1e-6).astype(np.float32)[None, :]
    for b, n, y in zip(blocks, shapes, ys):
        _check(y, oracle.q4k_matvec(b, K, n, xn))


@pytest.mark.parametrize("fmt", [12, 8])
@pytest.mark.parametrize("K,N,M", [(2560, 10240, 16), (2560, 300, 33), (10240, 2560, 64),
                                   (256, 1, 17), (512, 129, 100), (2560, 2048, 256)])
def test_batched_tensor_core_path(ctx, oracle, fmt, K, N, M):
    """16 or more tokens: weights dequantised to f16 into the context's arena, product on
    tcgen05 (kind::f16) with the activations split hi + lo.  Same 1e-3 bar; the f16 rounding
    of the weights puts this path near 3e-4."""
    rng = np.random.default_rng(K + N + M + fmt)
    blocks = formats.random_kquant(rng, fmt, N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    gamma = (1.0 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    res = rng.standard_normal((M, N)).astype(np.float32)
    layer = LinearLayer.create_from_bytes(ctx, blocks, fmt, K, N)
    rows = sorted(set([0, M // 2, M - 1]))  # the f64 oracle is slow: check three tokens
    y = layer.forward(_dev(x), residual=_dev(res))
    ctx.check()
    ref = oracle.kquant_matvec(fmt, blocks, K, N, x[rows], residual=res[rows])
    _check(y[rows], ref)
    xn = np.stack([oracle.rmsnorm_f64(x[m], gamma, 1e-6) for m in rows]).astype(np.float32)
    y = layer.forward(_dev(x), rms_gamma=_dev(gamma), eps=1e-6)
    ctx.check()
    _check(y[rows], oracle.kquant_matvec(fmt, blocks, K, N, xn))


@pytest.mark.parametrize("fmt", [12, 8])
def test_batched_path_over_the_f16_range(ctx, oracle, fmt):
    """The tensor-core path rounds activations to f16, whose largest finite value is 65504: a
    FFN intermediate of a few 1e4 is ordinary.  Every staged row is scaled by its own power of
    two, so rows of magnitude 1e-6, 1, 3e4 and 1e6 in one call all meet the 1e-3 bar, also
    through the gate/up GLU epilogue (per row the same bar as for unit-magnitude inputs)."""
    K, N, M = 2560, 384, 20
    rng = np.random.default_rng(500 + fmt)
    blocks = formats.random_kquant(rng, fmt, N, K)
    mags = np.array([1e-6, 1.0, 3e4, 1e6], np.float32)[np.arange(M) % 4]
    x = (rng.standard_normal((M, K)) * mags[:, None]).astype(np.float32)
    layer = LinearLayer.create_from_bytes(ctx, blocks, fmt, K, N)
    y = layer.forward(_dev(x)).cpu().numpy()
    ctx.check()
    ref = oracle.kquant_matvec(fmt, blocks, K, N, x)
    assert np.isfinite(y).all()
    for m in range(M):
        assert np.max(np.abs(y[m] - ref[m])) <= TOL * np.max(np.abs(ref[m])), (m, mags[m])
    if fmt == 12:
        up = formats.random_kquant(rng, fmt, N, K)
        lu = LinearLayer.create_from_bytes(ctx, up, fmt, K, N)
        xs = (rng.standard_normal((M, K)) * np.minimum(mags, 30.0)[:, None]).astype(np.float32)
        g = LinearLayer.forward_fused_gate_up(layer, lu, _dev(xs)).cpu().numpy()
        ctx.check()
        gref = oracle.kquant_gateup_gelu(blocks, up, fmt, K, N, xs)
        assert np.isfinite(g).all()
        for m in range(M):
            assert np.max(np.abs(g[m] - gref[m])) <= 2e-3 * np.max(np.abs(gref[m])), (m, mags[m])


def test_batched_row_chunks_of_the_arena(ctx, oracle):
    # 2560 x 16384 f16 = 80 MB: more than the 64 MB arena, so two row chunks
    K, N, M = 2560, 16384, 20
    rng = np.random.default_rng(77)
    blocks = formats.random_q4k(rng, N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    y = LinearLayer.create_from_bytes(ctx, blocks, 12, K, N).forward(_dev(x))
    ctx.check()
    _check(y[[0, 19]], oracle.q4k_matvec(blocks, K, N, x[[0, 19]]))


@pytest.mark.parametrize("K,N,M", [(2560, 1000, 16), (2560, 1000, 70), (2560, 1000, 256),
                                   (512, 9000, 200), (10240, 640, 150)])
def test_batched_gate_up_and_multi(ctx, oracle, K, N, M):
    """Gate and up share one staging of the activations; the GLU is the up product's epilogue
    (with and without split-K, 64 / 128 / 256 tokens per pass, several passes)."""
    rng = np.random.default_rng(M)
    bg = formats.random_q4k(rng, N, K)
    bu = formats.random_q4k(rng, N, K)
    x = rng.standard_normal((M, K)).astype(np.float32)
    g = LinearLayer.create_from_bytes(ctx, bg, 12, K, N)
    u = LinearLayer.create_from_bytes(ctx, bu, 12, K, N)
    y = LinearLayer.forward_fused_gate_up(g, u, _dev(x))
    ctx.check()
    rows = [0, M - 1]
    # gelu(gate) * up is a PRODUCT of two k-quant outputs: on the tensor-core path each factor
    # carries the f16 rounding of its weights and activations (~4e-4 of its own scale, inside
    # the 1e-3 bar, checked on ys below), so the product is held to twice the bar
    _check(y[rows], oracle.kquant_gateup_gelu(bg, bu, 12, K, N, x[rows]), tol=2e-3)
    ys = LinearLayer.forward_multi([g, u], _dev(x))
    ctx.check()
    _check(ys[0][rows], oracle.q4k_matvec(bg, K, N, x[rows]))
    _check(ys[1][rows], oracle.q4k_matvec(bu, K, N, x[rows]))


@pytest.mark.parametrize("fmt", [12, 8])
@pytest.mark.parametrize("M", [1, 3, 20])
def test_post_norm_folded_into_the_next_matvec(ctx, oracle, fmt, M):
    """x' = base + rmsnorm(o) * g1 in front of a fused-norm q/k/v call and of a gate/up call:
    x' and the products equal the oracle's evaluation of the same chain (streaming kernel's
    prologue for M < 16, separate launch in front of the tensor-core path from 16 on)."""
    K, N = 2560, 384
    rng = np.random.default_rng(100 + M + fmt)
    ba = formats.random_kquant(rng, fmt, N, K)
    bb = formats.random_kquant(rng, fmt, N, K)
    o = rng.standard_normal((M, K)).astype(np.float32)
    base = rng.standard_normal((M, K)).astype(np.float32)
    g1 = (1.0 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    g2 = (1.0 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    la = LinearLayer.create_from_bytes(ctx, ba, fmt, K, N)
    lb = LinearLayer.create_from_bytes(ctx, bb, fmt, K, N)
    xp = np.stack([base[m].astype(np.float64) + oracle.rmsnorm_f64(o[m], g1, 1e-6)
                   for m in range(M)])
    xn = np.stack([oracle.rmsnorm_f64(xp[m].astype(np.float32), g2, 1e-6)
                   for m in range(M)]).astype(np.float32)
    do, dbase, dg1, dg2 = _dev(o), _dev(base), _dev(g1), _dev(g2)
    ys, xo = LinearLayer.forward_multi([la, lb], do, rms_gamma=dg2, eps=1e-6, pre=(dbase, dg1))
    ctx.check()
    assert np.max(np.abs(xo.cpu().numpy() - xp)) <= 1e-5 * np.max(np.abs(xp))
    _check(ys[0], oracle.kquant_matvec(fmt, ba, K, N, xn))
    _check(ys[1], oracle.kquant_matvec(fmt, bb, K, N, xn))
    y, xo2 = LinearLayer.forward_fused_gate_up(la, lb, do, rms_gamma=dg2, eps=1e-6,
                                               pre=(dbase, dg1))
    ctx.check()
    assert torch.equal(xo, xo2)
    # one token and three take the streaming kernels (1e-3 holds for the product too); 20
    # tokens take the f16 tensor-core path, where the product of two outputs gets twice the bar
    _check(y, oracle.kquant_gateup_gelu(ba, bb, fmt, K, N, xn), tol=TOL if M < 16 else 2e-3)
    # and the unfused sequence of calls gives the same x' bit for bit
    ref = LinearLayer.forward_multi([la, lb], xo, rms_gamma=dg2, eps=1e-6)
    ctx.check()
    _check(ys[0], ref[0].cpu().numpy(), tol=1e-6)


@pytest.mark.parametrize("fmt", [12, 8])
def test_linearity_full_size(ctx, fmt):
    """Size-independent property at the benchmark shape: y(a*x) = a*y(x) for a power of two
    (the block quantiser scales exactly), and zero input gives zero output."""
    K, N = 2560, 10240
    rng = np.random.default_rng(21)
    layer = LinearLayer.create_from_bytes(ctx, formats.random_kquant(rng, fmt, N, K), fmt, K, N)
    x = _dev(rng.standard_normal((1, K)).astype(np.float32))
    y1 = layer.forward(x)
    y4 = layer.forward(x * 4.0)
    assert torch.equal(y4, y1 * 4.0)
    assert not layer.forward(torch.zeros_like(x)).any()
    assert torch.equal(layer.forward(x), y1)  # deterministic


# ---- the mma.sync one-token kernel, forced on at every shape that fits (ctx_mv) -------------

@pytest.mark.parametrize("fmt", [12, 8])
@pytest.mark.parametrize("K,N", [(2560, 10240), (2560, 2048), (2048, 2560), (10240, 2560),
                                 (256, 1), (512, 7), (768, 33), (4096, 1000), (1280, 2560)])
def test_mv_kernel_shapes(ctx_mv, oracle, fmt, K, N):
    """Ragged last tiles, fewer super-blocks than warps (K < 2560), several per warp (K = 10240),
    one row, with residual and with the RMSNorm prologue."""
    rng = np.random.default_rng(5 * K + N + fmt)
    blocks = formats.random_kquant(rng, fmt, N, K)
    x = rng.standard_normal((1, K)).astype(np.float32)
    res = rng.standard_normal((1, N)).astype(np.float32)
    gamma = (1.0 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    layer = LinearLayer.create_from_bytes(ctx_mv, blocks, fmt, K, N)
    def check(y, ref, design=None):
        if N >= 4:
            err = _check(y, ref)
            assert design is None or err < design
        else:  # a single output can cancel to almost nothing: measure against the terms' size
            assert np.max(np.abs(y.cpu().numpy() - ref)) <= 1e-3 * np.sqrt(K) * 0.3

    check(layer.forward(_dev(x), residual=_dev(res)),
          oracle.kquant_matvec(fmt, blocks, K, N, x, residual=res), design=2e-4)
    xn = oracle.rmsnorm_f64(x[0], gamma, 1e-6).astype(np.float32)[None, :]
    check(layer.forward(_dev(x), rms_gamma=_dev(gamma), eps=1e-6),
          oracle.kquant_matvec(fmt, blocks, K, N, xn))
    ctx_mv.check()


@pytest.mark.parametrize("fmt", [12, 8])
def test_mv_kernel_matches_streaming_kernel_on_heavy_tails(ctx, ctx_mv, oracle, fmt):
    """Activations with outliers 100x the typical size: the per-32 block scales keep both
    kernels inside the bar."""
    K, N = 2560, 640
    rng = np.random.default_rng(31 + fmt)
    blocks = formats.random_kquant(rng, fmt, N, K)
    x = rng.standard_normal((1, K)).astype(np.float32)
    x[0, rng.integers(0, K, 12)] *= 100.0
    ref = oracle.kquant_matvec(fmt, blocks, K, N, x)
    _check(LinearLayer.create_from_bytes(ctx_mv, blocks, fmt, K, N).forward(_dev(x)), ref)
    _check(LinearLayer.create_from_bytes(ctx, blocks, fmt, K, N).forward(_dev(x)), ref)


@pytest.mark.parametrize("fmt", [12, 8])
def test_mv_kernel_fused_paths(ctx_mv, oracle, fmt):
    """q/k/v in one launch (rows of a CTA straddle tensors), gate/up GELU (tiles of 8 + 8 rows),
    and the folded post-norm in front of both."""
    K = 2560
    rng = np.random.default_rng(9 + fmt)
    shapes = [2048, 520, 504]
    blocks = [formats.random_kquant(rng, fmt, n, K) for n in shapes]
    x = rng.standard_normal((1, K)).astype(np.float32)
    gamma = (1.0 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    layers = [LinearLayer.create_from_bytes(ctx_mv, b, fmt, K, n) for b, n in zip(blocks, shapes)]
    ys = LinearLayer.forward_multi(layers, _dev(x), rms_gamma=_dev(gamma), eps=1e-6)
    xn = oracle.rmsnorm_f64(x[0], gamma, 1e-6).astype(np.float32)[None, :]
    for b, n, y in zip(blocks, shapes, ys):
        _check(y, oracle.kquant_matvec(fmt, b, K, n, xn))
    for N in (10240, 1000, 8):
        bg = formats.random_kquant(rng, fmt, N, K)
        bu = formats.random_kquant(rng, fmt, N, K)
        g = LinearLayer.create_from_bytes(ctx_mv, bg, fmt, K, N)
        u = LinearLayer.create_from_bytes(ctx_mv, bu, fmt, K, N)
        _check(LinearLayer.forward_fused_gate_up(g, u, _dev(x)),
               oracle.kquant_gateup_gelu(bg, bu, fmt, K, N, x))
    # folded post-norm: x' = base + rmsnorm(o) * g1, then RMSNorm(g2) and the products
    N = 384
    ba = formats.random_kquant(rng, fmt, N, K)
    bb = formats.random_kquant(rng, fmt, N, K)
    o = rng.standard_normal((1, K)).astype(np.float32)
    base = rng.standard_normal((1, K)).astype(np.float32)
    g1 = (1.0 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    la = LinearLayer.create_from_bytes(ctx_mv, ba, fmt, K, N)
    lb = LinearLayer.create_from_bytes(ctx_mv, bb, fmt, K, N)
    xp = base[0].astype(np.float64) + oracle.rmsnorm_f64(o[0], g1, 1e-6)
    xn = oracle.rmsnorm_f64(xp.astype(np.float32), gamma, 1e-6).astype(np.float32)[None, :]
    ys, xo = LinearLayer.forward_multi([la, lb], _dev(o), rms_gamma=_dev(gamma), eps=1e-6,
                                       pre=(_dev(base), _dev(g1)))
    assert np.max(np.abs(xo.cpu().numpy()[0] - xp)) <= 1e-5 * np.max(np.abs(xp))
    _check(ys[0], oracle.kquant_matvec(fmt, ba, K, N, xn))
    _check(ys[1], oracle.kquant_matvec(fmt, bb, K, N, xn))
    y, xo2 = LinearLayer.forward_fused_gate_up(la, lb, _dev(o), rms_gamma=_dev(gamma), eps=1e-6,
                                               pre=(_dev(base), _dev(g1)))
    assert torch.equal(xo, xo2)
    _check(y, oracle.kquant_gateup_gelu(ba, bb, fmt, K, N, xn))
    ctx_mv.check()


def test_mv_kernel_deterministic_and_linear(ctx_mv):
    K, N = 2560, 10240
    rng = np.random.default_rng(22)
    layer = LinearLayer.create_from_bytes(ctx_mv, formats.random_q4k(rng, N, K), 12, K, N)
    x = _dev(rng.standard_normal((1, K)).astype(np.float32))
    y1 = layer.forward(x)
    assert torch.equal(layer.forward(x), y1)
    assert torch.equal(layer.forward(x * 4.0), y1 * 4.0)
    assert not layer.forward(torch.zeros_like(x)).any()


def test_bad_arguments(ctx):
    from hesper_b200 import HesperB200Error
    layer = LinearLayer.create_from_bytes(ctx, np.zeros(144, np.uint8), 12, 256, 1)
    layer.in_dim = 128
    with pytest.raises(HesperB200Error):
        layer.forward(torch.zeros(1, 128, device="cuda"))
