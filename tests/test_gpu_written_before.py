"""Operands that a call reads ahead of its turn (launches overlap), written by the calls just before it."""
import numpy as np
import pytest

from oracle import cpu
from helpers import check_close, make_weight, make_x

pytestmark = pytest.mark.gpu


def _f16(ctx, buf, shape):
    return ctx.download(buf, shape, np.uint16).view(np.float16)


def _poison(ctx, buf, nbytes):
    ctx.L.nn_buf_fill(ctx.h, buf, 0x7E, nbytes)


def _producers(nnb, ctx, T, H):
    """Calls that write T x H values: a GEMM and, where that is one row, the streaming kernel; with their expected results."""
    M = T if T > 1 else 1
    x = make_x(M, H, 81)
    W, _ = make_weight("fp16", H, H, 82)
    q = nnb.QuantWeight(ctx, "fp16", W, None)
    xb = ctx.upload(x.view(np.uint16))

    def call(out):
        ctx.linear(M, H, H, xb, q.buf, out)

    def free():
        q.release()
        ctx.free(xb)

    return call, x.astype(np.float64) @ W.astype(np.float64).T, free


def test_norm_weight(nnb, ctx):
    rows, cols = 64, 4096
    call, want_g, free = _producers(nnb, ctx, 1, cols)
    x = make_x(rows, cols, 83)
    xb, g, out = ctx.upload(x.view(np.uint16)), ctx.alloc(cols * 2), ctx.alloc(rows * cols * 2)
    for _ in range(4):
        _poison(ctx, g, cols * 2)
        call(g)
        ctx.rmsnorm(rows, cols, xb, g, 1e-5, out)
        got_g = _f16(ctx, g, (cols,))
        check_close(got_g, want_g[0], what="norm weight")
        check_close(_f16(ctx, out, (rows, cols)), cpu.rmsnorm(x, got_g, 1e-5), what="norm with a weight just written")
    free()
    for b in (xb, g, out):
        ctx.free(b)


@pytest.mark.parametrize("between", [0, 6])
def test_gemm_weight(nnb, ctx, between):
    """Keys projected from a prompt, any number of small calls, then scores against the keys."""
    M, T, H = 48, 640, 512
    call, want_k, free = _producers(nnb, ctx, T, H)
    x = make_x(M, H, 91)
    W, _ = make_weight("fp16", 64, H, 92)
    q = nnb.QuantWeight(ctx, "fp16", W, None)
    xb, keys, out = ctx.upload(x.view(np.uint16)), ctx.alloc(T * H * 2), ctx.alloc(M * T * 2)
    small = [[ctx.alloc(M * 64 * 2) for _ in range(3)] for _ in range(between)]
    for _ in range(4):
        _poison(ctx, keys, T * H * 2)
        call(keys)
        for o in small:
            ctx.linear_qkv(M, H, xb, q.buf, 64, q.buf, 64, q.buf, 64, *o)
        ctx.linear(M, T, H, xb, keys, out)
        k = _f16(ctx, keys, (T, H)).astype(np.float64)
        check_close(k, want_k, what="projected keys")
        check_close(_f16(ctx, out, (M, T)), x.astype(np.float64) @ k.T, what=f"scores, {between} calls between")
    free()
    q.release()
    for b in [xb, keys, out] + sum(small, []):
        ctx.free(b)
