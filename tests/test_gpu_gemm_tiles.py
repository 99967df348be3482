"""The tensor-core GEMM (M > 16) where its tiling can go wrong: row and token tiles with remainders, K tails of every
format (short packed spans included), outputs whose rows are not 16-byte aligned, tiles split over a cluster, every
epilogue, and a weight that the call before has just written; and the row-wise RMSNorm in front of it."""
import numpy as np
import pytest

from oracle import cpu
from helpers import alloc_with_canary, check_canary, check_close, make_weight, make_x

pytestmark = pytest.mark.gpu


def _want(fmt, x, W, s):
    return x.astype(np.float64) @ cpu.dequant(fmt, W, s).astype(np.float64).T


def _silu(v):
    return v / (1.0 + np.exp(-v))


# (N, K, M): one row tile and one more row; 16 rows past a token tile; K of one block, of one and a half spans, of many spans
# over a cluster; the widest token tile with a remainder; odd N (unaligned rows)
SHAPES = [(128, 64, 17), (129, 64, 32), (127, 96, 33), (1000, 544, 80), (257, 1088, 49), (896, 4864, 40), (640, 992, 257), (1001, 2048, 100), (64, 8192, 20)]


@pytest.mark.parametrize("fmt", ["fp16", "int8", "q4"])
@pytest.mark.parametrize("N,K,M", SHAPES)
def test_tiles_and_epilogues(nnb, ctx, fmt, N, K, M):
    x, r = make_x(M, K, 31), make_x(M, N, 32)
    (W, s), (W2, s2) = make_weight(fmt, N, K, 33), make_weight(fmt, N, K, 34)
    q, q2 = nnb.QuantWeight(ctx, fmt, W, s), nnb.QuantWeight(ctx, fmt, W2, s2)
    xb, ob = ctx.upload(x.view(np.uint16)), alloc_with_canary(ctx, M * N * 2)
    y, y2 = _want(fmt, x, W, s), _want(fmt, x, W2, s2)
    r64 = r.astype(np.float64)

    def out():
        check_canary(ctx, ob, M * N * 2, f"{fmt} {N}x{K} M={M}")
        return ctx.download(ob, (M, N), np.uint16).view(np.float16)

    ctx.linear(M, N, K, xb, q.buf, ob)
    check_close(out(), y, what=f"store {fmt} {N}x{K} M={M}")
    ctx.fused_gate_up_silu(M, N, K, xb, q.buf, q2.buf, ob)
    check_close(out(), _silu(y) * y2, what=f"swiglu {fmt} {N}x{K} M={M}")
    ctx.upload(r.view(np.uint16), ob)
    ctx.linear_add(M, N, K, xb, q.buf, ob)
    check_close(out(), r64 + y, what=f"residual {fmt} {N}x{K} M={M}")
    ctx.upload(r.view(np.uint16), ob)
    ctx.linear_silu_gate_fused(M, N, K, xb, q.buf, ob)
    check_close(out(), _silu(r64) * y, what=f"silu gate {fmt} {N}x{K} M={M}")
    for w in (q, q2):
        w.release()
    for b in (xb, ob):
        ctx.free(b)


@pytest.mark.parametrize("fmt", ["fp16", "int8", "q4"])
def test_pairs_of_blocks(nnb, ctx, fmt):
    """Enough tiles for two blocks on each: an odd number of row tiles, remainders in rows, tokens and K."""
    M, N, K = 1000, 128 * 146 + 8, 544
    x, r = make_x(M, K, 61), make_x(M, N, 62)
    (W, s), (W2, s2) = make_weight(fmt, N, K, 63), make_weight(fmt, N, K, 64)
    q, q2 = nnb.QuantWeight(ctx, fmt, W, s), nnb.QuantWeight(ctx, fmt, W2, s2)
    xb, ob = ctx.upload(x.view(np.uint16)), alloc_with_canary(ctx, M * N * 2)
    y, y2 = _want(fmt, x, W, s), _want(fmt, x, W2, s2)
    ctx.upload(r.view(np.uint16), ob)
    ctx.linear_add(M, N, K, xb, q.buf, ob)
    check_close(ctx.download(ob, (M, N), np.uint16).view(np.float16), r.astype(np.float64) + y, what=f"residual {fmt}")
    ctx.fused_gate_up_silu(M, N, K, xb, q.buf, q2.buf, ob)
    check_close(ctx.download(ob, (M, N), np.uint16).view(np.float16), _silu(y) * y2, what=f"swiglu {fmt}")
    check_canary(ctx, ob, M * N * 2, fmt)
    for w in (q, q2):
        w.release()
    for b in (xb, ob):
        ctx.free(b)


@pytest.mark.parametrize("fmt", ["fp16", "int8", "q4"])
@pytest.mark.parametrize("M,Ns", [(33, (200, 72, 65)), (600, (896, 128, 128))])
def test_three_weights_with_bias(nnb, ctx, fmt, M, Ns):
    """One launch over three weights of unequal, unaligned row counts: one row tile of each, and several of one beside one."""
    K = 448
    x = make_x(M, K, 41)
    ws = [make_weight(fmt, n, K, 42 + i) for i, n in enumerate(Ns)]
    bs = [make_x(1, n, 45 + i)[0] for i, n in enumerate(Ns)]
    qs = [nnb.QuantWeight(ctx, fmt, W, s) for W, s in ws]
    xb = ctx.upload(x.view(np.uint16))
    bb = [ctx.upload(b.view(np.uint16)) for b in bs]
    outs = [alloc_with_canary(ctx, M * n * 2) for n in Ns]
    ctx.linear_qkv_bias(M, K, xb, qs[0].buf, Ns[0], qs[1].buf, Ns[1], qs[2].buf, Ns[2], *bb, *outs)
    for (W, s), b, o, n in zip(ws, bs, outs, Ns):
        want = _want(fmt, x, W, s).astype(np.float16).astype(np.float32) + b.astype(np.float32)[None, :]
        check_close(ctx.download(o, (M, n), np.uint16).view(np.float16), want, what=f"qkv bias {fmt} M={M} N={n}")
        check_canary(ctx, o, M * n * 2, f"qkv bias {fmt} M={M} N={n}")
    for w in qs:
        w.release()
    for b in [xb] + bb + outs:
        ctx.free(b)


@pytest.mark.parametrize("N", [4096, 2051])
def test_swiglu_has_the_bits_of_few_rows(nnb, ctx, N):
    """One-hot activations: gate and up are single weights, exact in both kernels, and what is left is SiLU(gate) * up.  Gates: at
    N = 4096 every fp16 value, infinities and NaNs too, with ups of every magnitude; else the usual range."""
    M, K = 64, 64
    rng = np.random.default_rng(65)
    if N * K == 1 << 18:
        # column m of the weights holds the values of row m; rows of x pick one column, so no infinity meets a zero of another
        Wg = np.tile(np.arange(1 << 16, dtype=np.uint16), 4).reshape(K, N)
        Wu = rng.integers(0, 0x7C00, (K, N)).astype(np.uint16) | (rng.integers(0, 2, (K, N)) << 15).astype(np.uint16)
        Wg, Wu = Wg.view(np.float16), Wu.view(np.float16)
    else:
        Wg, Wu = rng.uniform(-14.0, 14.0, (K, N)).astype(np.float16), rng.standard_normal((K, N)).astype(np.float16)
    special = ~np.isfinite(Wg.astype(np.float32))
    xb, ob = ctx.upload(np.eye(M, K, dtype=np.float16).view(np.uint16)), ctx.alloc(M * N * 2)

    def both(wg):
        qg, qu = (nnb.QuantWeight(ctx, "fp16", np.ascontiguousarray(w.T), None) for w in (wg, Wu))
        ctx.fused_gate_up_silu(M, N, K, xb, qg.buf, qu.buf, ob)
        many = ctx.download(ob, (M, N), np.uint16)
        few = []
        for m in range(0, M, 16):
            ctx.fused_gate_up_silu(16, N, K, xb + m * K * 2, qg.buf, qu.buf, ob)
            few.append(ctx.download(ob, (16, N), np.uint16))
        qg.release()
        qu.release()
        return many, np.concatenate(few)

    finite = np.where(special, np.float16(0), Wg)
    many, few = both(finite)
    assert np.array_equal(many, few), f"{(many != few).sum()} of {many.size} values"
    g, u = finite.astype(np.float64), Wu.astype(np.float64)
    with np.errstate(over="ignore"):
        want = (g / (1.0 + np.exp(-g)) * u).astype(np.float16)
    got = many.view(np.float16)
    near = np.isfinite(want) & np.isfinite(got)
    assert (~near).sum() == (~np.isfinite(want)).sum() == (~np.isfinite(got)).sum()
    check_close(got[near], want[near], what="swiglu of single weights")
    if special.any():   # a whole column of them, so that every row meets one: an infinity times zero is a NaN in both kernels
        many, few = both(np.where(special, Wg, np.float16(1)))
        nan = np.isnan(few.view(np.float16))
        assert np.array_equal(np.isnan(many.view(np.float16)), nan) and np.array_equal(many[~nan], few[~nan])
    for b in (xb, ob):
        ctx.free(b)


def test_weight_written_by_the_call_before(nnb, ctx):
    """A weight may be another call's result (scores against keys just projected): nothing of it is fetched early."""
    M, T, H = 48, 640, 512
    x, k_in = make_x(M, H, 51), make_x(T, H, 52)
    Wk, _ = make_weight("fp16", H, H, 53)
    q = nnb.QuantWeight(ctx, "fp16", Wk, None)
    xb, kb, keys, out = ctx.upload(x.view(np.uint16)), ctx.upload(k_in.view(np.uint16)), ctx.alloc(T * H * 2), ctx.alloc(M * T * 2)
    for _ in range(4):
        ctx.L.nn_buf_fill(ctx.h, keys, 0x7e, T * H * 2)
        ctx.linear(T, H, H, kb, q.buf, keys)
        ctx.linear(M, T, H, xb, keys, out)
        k = ctx.download(keys, (T, H), np.uint16).view(np.float16).astype(np.float64)
        check_close(ctx.download(out, (M, T), np.uint16).view(np.float16), x.astype(np.float64) @ k.T, what="x . (projected keys)^T")
    q.release()
    for b in (xb, kb, keys, out):
        ctx.free(b)


@pytest.mark.parametrize("rows,cols", [(1, 8), (5, 256), (33, 2048), (7, 2056), (4, 4864), (3, 100)])
def test_rmsnorm_rows(nnb, ctx, rows, cols):
    x = (make_x(rows, cols, 61).astype(np.float32) * 3.0).astype(np.float16)
    g = (1.0 + 0.1 * np.random.default_rng(62).standard_normal(cols)).astype(np.float16)
    dx, dg, out = ctx.upload(x.view(np.uint16)), ctx.upload(g.view(np.uint16)), alloc_with_canary(ctx, rows * cols * 2)
    ctx.rmsnorm(rows, cols, dx, dg, 1e-5, out)
    check_close(ctx.download(out, (rows, cols), np.uint16).view(np.float16), cpu.rmsnorm(x, g, 1e-5), what=f"rmsnorm {rows}x{cols}")
    check_canary(ctx, out, rows * cols * 2, f"rmsnorm {rows}x{cols}")
    for b in (dx, dg, out):
        ctx.free(b)
