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


@pytest.mark.parametrize("M", [1, 5, 40])
@pytest.mark.parametrize("fmt", ["fp16", "int8"])
def test_bias(nnb, ctx, fmt, M):
    K, Ns = 896, (896, 128, 128)
    call, want_b, free = _producers(nnb, ctx, 1, 896)
    x = make_x(M, K, 84)
    ws = [make_weight(fmt, n, K, 85 + i) for i, n in enumerate(Ns)]
    qs = [nnb.QuantWeight(ctx, fmt, W, s) for W, s in ws]
    xb, bias = ctx.upload(x.view(np.uint16)), ctx.alloc(896 * 2)
    outs = [ctx.alloc(M * n * 2) for n in Ns]
    for _ in range(4):
        _poison(ctx, bias, 896 * 2)
        call(bias)
        ctx.linear_qkv_bias(M, K, xb, qs[0].buf, Ns[0], qs[1].buf, Ns[1], qs[2].buf, Ns[2], bias, bias, bias, *outs)
        b = _f16(ctx, bias, (896,))
        check_close(b, want_b[0], what="bias")
        for (W, s), o, n in zip(ws, outs, Ns):
            y = (x.astype(np.float64) @ cpu.dequant(fmt, W, s).astype(np.float64).T).astype(np.float16).astype(np.float32)
            check_close(_f16(ctx, o, (M, n)), y + b[:n].astype(np.float32), what=f"{fmt} M={M} bias just written")
    free()
    for q in qs:
        q.release()
    for b in [xb, bias] + outs:
        ctx.free(b)


@pytest.mark.parametrize("T", [1, 7, 640])
def test_weight_of_a_single_row(nnb, ctx, T):
    """One row against keys that a GEMM, a batched or a single-row call has just written."""
    H = 512
    call, want_k, free = _producers(nnb, ctx, T, H)
    x = make_x(1, H, 93)
    xb, keys, out, tok = ctx.upload(x.view(np.uint16)), ctx.alloc(T * H * 2), ctx.alloc(T * 2), ctx.alloc(4)
    for _ in range(4):
        for pick in (False, True):
            _poison(ctx, keys, T * H * 2)
            call(keys)
            if pick:
                ctx.linear_argmax(T, H, xb, keys, out, tok)
            else:
                ctx.linear(1, T, H, xb, keys, out)
            k = _f16(ctx, keys, (T, H)).astype(np.float64)
            check_close(k, want_k, what="projected keys")
            check_close(_f16(ctx, out, (T,)), (x.astype(np.float64) @ k.T)[0], what=f"scores of one row against {T} keys")
    free()
    for b in (xb, keys, out, tok):
        ctx.free(b)


@pytest.mark.parametrize("which", ["weight", "norm", "bias"])
def test_recorded_step(nnb, ctx, which):
    """The same inside a recording: the operator is no part of a resident run, and a replay has the results of the calls."""
    H = 512
    W, _ = make_weight("fp16", H, H, 94)
    q = nnb.QuantWeight(ctx, "fp16", W, None)
    x, g = make_x(1, H, 95), make_x(1, H, 96)
    xb, gb = ctx.upload(x.view(np.uint16)), ctx.upload(g.view(np.uint16))
    a, b, made, out = (ctx.alloc(H * 2) for _ in range(4))
    o3 = [ctx.alloc(H * 2) for _ in range(3)]

    def step():
        ctx.linear(1, H, H, xb, q.buf, a)
        ctx.linear(1, H, H, gb, q.buf, made)      # the weight (of one row), norm weight or bias that is used below
        ctx.linear(1, H, H, a, q.buf, b)
        if which == "weight":
            ctx.linear(1, 1, H, b, made, out)
        elif which == "norm":
            ctx.rmsnorm_linear(1, H, H, b, made, 1e-5, q.buf, out)
        else:
            ctx.linear_qkv_bias(1, H, b, q.buf, H, q.buf, H, q.buf, H, made, made, made, out, *o3[:2])
        ctx.linear(1, H, H, b, q.buf, o3[2])
        ctx.linear(1, H, H, o3[2], q.buf, a)

    n = 1 if which == "weight" else H
    for t in (a, b, made, out):
        _poison(ctx, t, H * 2)
    step()
    ctx.sync()
    eager = [ctx.download(t, (m,), np.uint16) for t, m in ((made, H), (out, n), (a, H))]
    assert np.isfinite(eager[1].view(np.float16)).all()
    ctx.plan_begin()
    step()
    plan = ctx.plan_end()
    for _ in range(3):
        for t in (a, b, made, out):
            _poison(ctx, t, H * 2)
        ctx.plan_launch(plan)
        ctx.sync()
        now = [ctx.download(t, (m,), np.uint16) for t, m in ((made, H), (out, n), (a, H))]
        assert all(np.array_equal(p, r) for p, r in zip(eager, now)), which
    assert ctx.L.nn_plan_num_kernels(plan) == 3      # two runs, and the operator between them
    ctx.L.nn_plan_free(plan)
    q.release()
    for t in [xb, gb, a, b, made, out] + o3:
        ctx.free(t)
