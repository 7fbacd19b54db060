"""Parity of the tcgen05 / TMEM projection kernel (taken for more than 64 tokens when the output width
is a multiple of 128 and K a multiple of 64) against the CPU oracle, and against the warp-level
kernel on the same inputs.  Same bounds as test_gpu_kernels.py: unrounded f32 accumulation within
2e-3, bf16 output within that plus its own rounding."""
import ctypes as C

import numpy as np
import pytest

from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    from mlx_llm_b200 import _lib, kernels
    from oracle import oracle as orc

    ctx = _lib.Context(0)
    yield ctx, kernels, orc, _lib
    ctx.close()


STREAM, RING, PAIR = 1, 2, 3  # kernels that K.projection names


def half_aligned(ctx, x):
    """The rows of x on the device at an address that is a multiple of 8 bytes, not of 16."""
    buf = ctx.buf(np.concatenate([np.zeros(4, np.uint16), x.ravel()]))
    half_aligned.alive = buf  # (until the next one)
    return buf.ptr + 8


def quant_case(seed, n, k, bits):
    rng = np.random.default_rng(seed)
    packed = rng.integers(0, 2**32, size=(n, k * bits // 32), dtype=np.uint32)
    s = np.abs(rng.standard_normal((n, k // 64)).astype(np.float32) * 0.02) / 7.5
    scales = H.f32_to_bf16_np(s)
    biases = H.f32_to_bf16_np(-8.0 * H.bf16_to_f32_np(scales) + rng.standard_normal((n, k // 64)).astype(np.float32) * 1e-3)
    return packed, scales, biases


@pytest.mark.parametrize("bits", [4, 8, 0])
@pytest.mark.parametrize("m,n,k", [(33, 256, 2048), (48, 384, 512), (64, 640, 1024), (65, 128, 64), (100, 256, 512), (256, 128, 4096), (300, 384, 1024), (700, 256, 2048),
                                   # more 256-token blocks than CTA pairs: several pieces per pair, two-block pieces,
                                   # a ragged last block, and an output width that is an odd multiple of 128
                                   (700, 20480, 256), (530, 19072, 128), (1100, 9984, 192)])
def test_tc_gemm_vs_oracle(env, bits, m, n, k):
    ctx, K, orc, _lib = env
    rng = np.random.default_rng(m + n + k)
    x = H.f32_to_bf16_np(rng.standard_normal((m, k)).astype(np.float32))
    dx = ctx.buf(x)
    yb, yf = ctx.empty((m, n), np.uint16), ctx.empty((m, n), np.float32)
    if bits:
        packed, scales, biases = quant_case(1, n, k, bits)
        K.qmm(ctx, dx, ctx.buf(packed), ctx.buf(scales), ctx.buf(biases), m, n, k, bits, yb, yf)
        rf, _ = orc.qmm(x, packed, scales, biases, 64, bits)
    else:
        w = H.f32_to_bf16_np(rng.standard_normal((n, k)).astype(np.float32) * 0.03)
        K.linear(ctx, dx, ctx.buf(w), m, n, k, yb, yf)
        rf, _ = orc.linear(x, w)
    ctx.sync()
    got = yf.download()
    assert np.isfinite(got).all()
    assert np.abs(got - rf).max() <= 2e-3, f"max-abs {np.abs(got - rf).max()}"
    assert H.close_bf16_out(yb.download(), rf)[0]


def test_tc_matches_warp_level_kernel(env):
    """Both projection kernels dequantise to the same bf16 weights and accumulate in f32: their
    unrounded outputs agree to f32 summation-order noise."""
    ctx, K, orc, _lib = env
    m, n, k = 512, 512, 4096
    rng = np.random.default_rng(0)
    x = H.f32_to_bf16_np(rng.standard_normal((m, k)).astype(np.float32))
    packed, scales, biases = quant_case(2, n, k, 4)
    dx, dp, ds, db = ctx.buf(x), ctx.buf(packed), ctx.buf(scales), ctx.buf(biases)
    outs = []
    for use_tc in (1, 0):
        _lib.check(_lib.load().b2_ctx_set_tensor_path(ctx.h, use_tc))
        y = ctx.empty((m, n), np.float32)
        K.qmm(ctx, dx, dp, ds, db, m, n, k, 4, None, y)
        ctx.sync()
        outs.append(y.download())
    _lib.check(_lib.load().b2_ctx_set_tensor_path(ctx.h, 1))
    assert np.abs(outs[0] - outs[1]).max() <= 1e-4


@pytest.mark.parametrize("bits", [4, 8, 0])
@pytest.mark.parametrize("m,n,k", [(1, 128, 256), (5, 256, 512), (8, 1024, 4096), (9, 128, 1024), (16, 384, 2048), (17, 256, 4096),
                                   (32, 512, 1024), (3, 128, 14336), (2, 256, 20480)])
def test_stream_gemm_vs_oracle(env, bits, m, n, k):
    """Up to 32 tokens with N a multiple of 128 and K of 256, quantized weights without a table of scales and biases or activations
    aligned to 8 bytes only, take the weight-streaming kernel: the token-tile counts 8, 16 and 32 wide, one and several K ranges, ragged
    token counts (from 33 tokens on the tcgen05 kernel takes every shape its tiling fits, see test_tc_gemm_vs_oracle)."""
    ctx, K, orc, _lib = env
    rng = np.random.default_rng(7 * m + n + k)
    x = H.f32_to_bf16_np(rng.standard_normal((m, k)).astype(np.float32))
    dx = ctx.buf(x) if bits else half_aligned(ctx, x)
    yb, yf = ctx.empty((m, n), np.uint16), ctx.empty((m, n), np.float32)
    if bits:
        packed, scales, biases = quant_case(3, n, k, bits)
        K.qmm(ctx, dx, ctx.buf(packed), ctx.buf(scales), ctx.buf(biases), m, n, k, bits, yb, yf)
        rf, _ = orc.qmm(x, packed, scales, biases, 64, bits)
    else:
        w = H.f32_to_bf16_np(rng.standard_normal((n, k)).astype(np.float32) * 0.03)
        dw = ctx.buf(w)
        assert K.projection(ctx, dx, dw, None, None, m, n, k, 0, y_f32=yf)[0] == STREAM
        K.linear(ctx, dx, dw, m, n, k, yb, yf)
        rf, _ = orc.linear(x, w)
    ctx.sync()
    got = yf.download()
    assert np.isfinite(got).all()
    assert np.abs(got - rf).max() <= 2e-3, f"max-abs {np.abs(got - rf).max()}"
    assert H.close_bf16_out(yb.download(), rf)[0]


def test_stream_matches_tile_kernel(env):
    """Same bf16 weights, f32 accumulation: the streaming kernel and the tile kernel agree to summation-order noise."""
    ctx, K, orc, _lib = env
    m, n, k = 7, 512, 4096
    rng = np.random.default_rng(1)
    x = H.f32_to_bf16_np(rng.standard_normal((m, k)).astype(np.float32))
    packed, scales, biases = quant_case(4, n, k, 4)
    dx, dp, ds, db = ctx.buf(x), ctx.buf(packed), ctx.buf(scales), ctx.buf(biases)
    outs = []
    for fast in (1, 0):
        _lib.check(_lib.load().b2_ctx_set_tensor_path(ctx.h, fast))
        y = ctx.empty((m, n), np.float32)
        K.qmm(ctx, dx, dp, ds, db, m, n, k, 4, None, y)
        ctx.sync()
        outs.append(y.download())
    _lib.check(_lib.load().b2_ctx_set_tensor_path(ctx.h, 1))
    assert np.abs(outs[0] - outs[1]).max() <= 1e-4


@pytest.mark.parametrize("m,n,k", [(1, 128, 256), (8, 128, 14336), (9, 2048, 2048), (16, 384, 7936), (17, 256, 512), (31, 1024, 2048), (3, 77824, 256),
                                   (32, 77824, 1024)])
def test_ring_gemm_vs_oracle(env, m, n, k):
    """Dense weights take the ring kernel up to 32 tokens: 8, 16 and 32 of them, one K range and several, more tiles than the machine
    holds at once (clusters of every size: test_ring_gives_the_streaming_kernels_bits)."""
    ctx, K, orc, _lib = env
    rng = np.random.default_rng(m + n + k)
    x = H.f32_to_bf16_np(rng.standard_normal((m, k)).astype(np.float32))
    w = H.f32_to_bf16_np(rng.standard_normal((n, k), dtype=np.float32) * np.float32(0.03))
    dx, dw = ctx.buf(x), ctx.buf(w)
    yb, yf = ctx.empty((m, n), np.uint16), ctx.empty((m, n), np.float32)
    assert K.projection(ctx, dx, dw, None, None, m, n, k, 0, y_f32=yf)[0] == RING
    K.linear(ctx, dx, dw, m, n, k, yb, yf)
    rf, _ = orc.linear(x, w)
    ctx.sync()
    assert np.abs(yf.download() - rf).max() <= 2e-3
    assert H.close_bf16_out(yb.download(), rf)[0]


# tokens, features, inputs, blocks per cluster, K ranges: every cluster size, one to four ranges a block, ranges of unequal length, one
# and several rounds of blocks
RING_PLANS = [(8, 128, 256, 1, 1), (5, 20480, 1024, 1, 2), (7, 20480, 2048, 1, 4), (2, 128, 1024, 2, 2), (16, 12288, 1536, 2, 3), (8, 128, 1536, 3, 3), (8, 6144, 3072, 3, 6),
              (13, 128, 2048, 4, 4), (8, 5120, 4096, 4, 8), (1, 128, 2560, 5, 5), (16, 128, 5120, 5, 10), (16, 128, 3072, 6, 6), (3, 128, 6144, 6, 12),
              (16, 128, 7168, 7, 14), (9, 128, 10240, 7, 20), (8, 128, 14336, 7, 28), (4, 128, 4096, 8, 8), (8, 128, 8192, 8, 16), (16, 128, 12288, 8, 24), (8, 128, 16384, 8, 32)]
WIDE_RING_PLANS = [(17, 128, 256, 1, 1), (32, 77824, 1024, 1, 1), (24, 128, 1024, 2, 2), (32, 128, 1536, 3, 3), (31, 128, 2048, 4, 4), (32, 128, 2560, 5, 5),
                   (18, 128, 3072, 6, 6), (32, 10240, 7168, 7, 7), (32, 128, 4096, 8, 8)]


@pytest.mark.parametrize("bits,plan", [(b, p) for b in (0, 4, 8) for p in RING_PLANS] + [(b, p) for b in (0, 8) for p in WIDE_RING_PLANS])
def test_ring_gives_the_streaming_kernels_bits(env, bits, plan):
    """The ring kernel, dense and with a table, sums in the order of the streaming kernel, in all three epilogues."""
    ctx, K, orc, _lib = env
    m, n, k, cluster, ranges = plan
    rng = np.random.default_rng(m * n + k + bits)
    x, h = (H.f32_to_bf16_np(rng.standard_normal(s).astype(np.float32)) for s in ((m, k), (m, n)))
    scales = biases = None
    if bits:
        packed, scales, biases = (ctx.buf(a) for a in quant_case(k, n, k, bits))
    else:  # sign and mantissa at random, exponents 2^-9 to 2^-6
        raw = rng.integers(0, 2**16, (n, k), dtype=np.uint16)
        packed = ctx.buf((raw & 0x807f) + ((118 + (raw >> 7 & 3)) << 7).astype(np.uint16))
    got = []
    for dx, kernel in ((ctx.buf(x), RING), (half_aligned(ctx, x), STREAM)):
        yb, yf, dh = ctx.empty((m, n), np.uint16), ctx.empty((m, n), np.float32), ctx.buf(h)
        for out in (dict(y_bf16=yb), dict(y_f32=yf), dict(h=dh)):
            route = K.projection(ctx, dx, packed, scales, biases, m, n, k, bits, **out)
            assert route == (kernel, int(bits > 0), ranges, cluster if kernel == RING else 0)
        ctx.sync()
        got.append([b.download((m, n)) for b in (yb, yf, dh)])
    assert np.isfinite(got[0][1]).all() and np.abs(got[0][1]).max() > 0.1
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("batch", [1, 8, 9, 16, 23])
def test_ring_gemm_quantized_in_a_model(env, bits, batch):
    """Quantized weights take the ring kernel where a model holds their table (Q4: up to 16 tokens): single-token steps of a small model
    against the oracle."""
    from mlx_llm_b200 import engine
    from tests.test_gpu_real_shapes import LLAMA_CUT, run_schedule

    ctx, K, orc, _lib = env
    cfg = dict(LLAMA_CUT, layers=1, hidden=512, heads=4, kv_heads=1, inter=2816, vocab=1024, quant_bits=bits)
    run_schedule((ctx, engine, K, orc), cfg, [[(i, 2 + i % 3) for i in range(batch)], [(i, 1) for i in range(batch)]])


def double_rounded(codes, scales, biases):
    """bf16(f32(code scale + bias)) and bf16(code scale + bias) as bits; [n, k] codes, [n, k / 64] scales and biases."""
    exact = codes.astype(np.float64) * np.repeat(H.bf16_to_f32_np(scales), 64, 1) + np.repeat(H.bf16_to_f32_np(biases), 64, 1)
    twice = H.f32_to_bf16_np(exact.astype(np.float32))
    # (the 52 bits of a double hold every sum here; odd behind the 16 bits of f32 that a bf16 drops: one rounding from there)
    word = exact.astype(np.float32).view(np.uint32)
    low = exact.astype(np.float32).astype(np.float64)
    toward_zero = word - ((np.abs(low) > np.abs(exact)) & (word & 0x7fffffff > 0)).astype(np.uint32)
    sticky = toward_zero | (low != exact).astype(np.uint32)
    return twice, H.f32_to_bf16_np(sticky.view(np.float32))


@pytest.mark.parametrize("m,kernel", [(8, RING), (16, RING), (32, RING), (512, PAIR)])
def test_q8_weights_are_rounded_as_dequantize_does(env, m, kernel):
    """Both kernels that read the table of scales and biases make the weights of b2_dequantize bit for bit, also where a bias far below
    its scale decides a tie: an identity matrix as activations reads the weights out."""
    ctx, K, orc, _lib = env
    n, k = 256, 512
    rng = np.random.default_rng(m)
    codes = rng.integers(0, 256, (n, k), dtype=np.uint8)
    mantissa = lambda: rng.integers(0, 128, (n, k // 64)) | rng.integers(0, 2, (n, k // 64)) << 15
    down = rng.integers(-20, 28, (n, k // 64))  # bits that the bias lies below the scale
    down[: n // 2] = np.clip(down[: n // 2], -20, 15)  # (row tiles without and with groups that are rounded twice)
    scales = (mantissa() | 116 << 7).astype(np.uint16)
    biases = (mantissa() | (116 - down) << 7).astype(np.uint16)
    biases[3::7, 1] = 0
    want, once = double_rounded(codes, scales, biases)
    assert (want != once)[n // 2:].sum() > 20 and (want == once)[: n // 2].all()
    packed = codes.view(np.uint32)
    plain = ctx.empty((n, k), np.uint16)
    dp, ds, db = ctx.buf(packed), ctx.buf(scales), ctx.buf(biases)
    K.dequantize(ctx, dp, ds, db, n, k, 8, plain)
    got = np.empty((n, k), np.uint16)
    for at in range(0, k, m):
        x = np.zeros((m, k), np.uint16)
        x[np.arange(m), at + np.arange(m)] = 0x3f80
        y = ctx.empty((m, n), np.uint16)
        route = K.projection(ctx, ctx.buf(x), dp, ds, db, m, n, k, 8, y_bf16=y)
        assert route[:2] == (kernel, 1)
        ctx.sync()
        got[:, at:at + m] = y.download().T
    zero = (got & 0x7fff == 0) & (want & 0x7fff == 0)
    assert ((got == want) | zero).all()
    assert ((plain.download() == want) | zero).all()


@pytest.mark.parametrize("rows", [32, 128])
def test_weights_that_the_call_before_wrote(env, rows):
    """A dense matrix that the projections in front have just written (by the ring kernel, by CTA pairs) is read whole by the ring
    kernel and, 8-byte aligned activations, by the streaming kernel."""
    ctx, K, orc, _lib = env
    n, k, inner = 128, 2048, 4096
    rng = np.random.default_rng(rows)
    normal = lambda *shape: H.f32_to_bf16_np(rng.standard_normal(shape).astype(np.float32))
    a, x = ctx.buf(normal(k, inner)), ctx.buf(normal(9, k))
    sources = [[ctx.buf(normal(rows, inner)) for _ in range(n // rows)] for _ in range(2)]
    w = ctx.buf(np.zeros((n, k), np.uint16))
    outs = [ctx.empty((8, n), np.float32) for _ in range(2)]
    want = []
    for turn in range(12):
        for at, source in enumerate(sources[turn & 1]):
            K.linear(ctx, source, a, rows, k, inner, y_bf16=w.ptr + at * rows * k * 2)
        x_at = x.ptr + (8 if turn & 2 else 0)  # (the streaming kernel, the ring kernel)
        K.linear(ctx, x_at, w, 8, n, k, y_f32=outs[0])
        ctx.sync()
        K.linear(ctx, x_at, w, 8, n, k, y_f32=outs[1])  # (nothing in flight any more)
        ctx.sync()
        want.append(outs[1].download())
        assert np.array_equal(outs[0].download(), want[-1])
    assert not np.array_equal(want[0], want[1]) and np.array_equal(want[0], want[4])


# exponents of scales and biases: lowest and highest; whether a table is possible; the size of the activations
TABLE_RANGES = {"ordinary": (-14, -8, True, 0), "smallest": (-133, -120, True, 0), "small_sums": (-30, -20, True, -90), "largest_unshifted": (-126, -6, True, 0),
                "shifted": (-125, -5, True, 0), "shifted_most": (-110, 10, True, 0), "too_large": (-8, 11, False, 0), "too_wide": (-111, 10, False, 0)}


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("m", [7, 64])
@pytest.mark.parametrize("name", TABLE_RANGES)
def test_table_of_any_size_of_scales(env, name, m, bits):
    """The kernels that read the scaled table give the bits of those that read scales and biases themselves, from subnormal scales to
    the largest that get a table, sums near the lower end of f32 too; matrices beyond take the other kernels."""
    ctx, K, orc, _lib = env
    lo, hi, possible, size = TABLE_RANGES[name]
    n, k = 256, 512
    rng = np.random.default_rng(m)

    def numbers():
        e = rng.integers(max(lo, -126), hi + 1, (n, k // 64))
        e[0, 0], e[1, 1] = hi, max(lo, -126)
        v = np.ldexp(1 + rng.integers(0, 128, e.shape) / 128, e) * rng.choice([-1.0, 1.0], e.shape)
        if lo < -126:
            v[2::3] = np.ldexp(rng.integers(1, 128, v[2::3].shape), -133)  # subnormal
        return H.f32_to_bf16_np(v.astype(np.float32))

    packed = rng.integers(0, 2**32, size=(n, k * bits // 32), dtype=np.uint32)
    scales, biases = numbers(), numbers()
    x = H.f32_to_bf16_np(np.ldexp(rng.standard_normal((m, k)), size).astype(np.float32))
    dx, dp, ds, db = ctx.buf(x), ctx.buf(packed), ctx.buf(scales), ctx.buf(biases)
    with_table, without = ctx.empty((m, n), np.float32), ctx.empty((m, n), np.float32)
    route = K.projection(ctx, dx, dp, ds, db, m, n, k, bits, y_f32=with_table)
    assert route[:2] == (PAIR if m > 32 else RING if possible else STREAM, int(possible))
    K.qmm(ctx, dx, dp, ds, db, m, n, k, bits, None, without)
    ctx.sync()
    want = without.download()
    assert np.isfinite(want).all() and np.abs(want).max() > 0
    assert np.array_equal(with_table.download(), want)
