"""Rows of an odd number of 32 values (int8, Q4): the second half of the last step lies past the row's end, where weights and activations are zeros."""
import numpy as np
import pytest

from helpers import alloc_with_canary, check_canary, check_close, make_weight, make_x
from oracle import cpu

pytestmark = pytest.mark.gpu


# tiles that split K (one chunk per quarter, several) and whole-row tiles, the shortest rows, rows too long to be resident for 16 rows
@pytest.mark.parametrize("fmt,N,K", [("int8", 100, 160), ("int8", 333, 736), ("int8", 70, 5152), ("int8", 40000, 352), ("int8", 64, 8224),
                                     ("q4", 100, 288), ("q4", 333, 736), ("q4", 70, 5152), ("q4", 40000, 352), ("int8", 40000, 5152)])
def test_rows(nnb, ctx, fmt, N, K):
    W, s = make_weight(fmt, min(N, 1000), K, 501)
    rep = -(-N // W.shape[0])
    Wn = np.tile(W, (rep, 1))[:N]
    sn = np.tile(s, (rep, 1) if s.ndim == 2 else rep)[:N]
    qw = nnb.QuantWeight(ctx, fmt, Wn, sn)
    x, r = make_x(16, K, 502), make_x(16, N, 503)
    x[4, :40] = np.float16(np.inf)      # (what lies behind row 3 in shared memory)
    good = [m for m in range(16) if m != 4]
    y = np.tile(x.astype(np.float64) @ cpu.dequant(fmt, W, s).astype(np.float64).T, (1, rep))[:, :N]
    xb, ob = ctx.upload(x.view(np.uint16)), alloc_with_canary(ctx, 16 * N * 2)
    ones = []
    for m in range(16):
        ctx.linear(1, N, K, xb + m * K * 2, qw.buf, ob + m * N * 2)
    ones = ctx.download(ob, (16, N), np.uint16).view(np.float16)
    check_close(ones[good], y[good], what=f"{fmt} {N}x{K}")
    for M in (3, 16):
        ctx.upload(r.view(np.uint16), ob)
        ctx.linear_add(M, N, K, xb, qw.buf, ob)
        got, rows = ctx.download(ob, (M, N), np.uint16).view(np.float16), [m for m in good if m < M]
        check_close(got[rows], r[rows].astype(np.float64) + y[rows], what=f"{fmt} {N}x{K} M={M} in place")
        ctx.linear(M, N, K, xb, qw.buf, ob)
        got = ctx.download(ob, (M, N), np.uint16).view(np.float16)
        check_close(got[rows], ones[rows], tol=2e-4, what=f"{fmt} {N}x{K} M={M} against single calls")
    ib = ctx.alloc(4)
    ctx.linear_argmax(N, K, xb, qw.buf, ob, ib)
    assert int(ctx.download(ib, (1,), np.int32)[0]) == cpu.argmax_half(ones[0])
    with pytest.raises(nnb.NNError):     # as before: a pick without logits wants rows of whole steps
        ctx.linear_argmax(N, K, xb, qw.buf, None, ib)
    check_canary(ctx, ob, 16 * N * 2, f"{fmt} {N}x{K}")
    qw.release()
    for b in (xb, ob, ib):
        ctx.free(b)


@pytest.mark.parametrize("fmt", ["int8", "q4"])
def test_recorded_run_and_fused_forms(nnb, ctx, fmt):
    K, F = 736, 1056
    ws = [nnb.QuantWeight(ctx, fmt, *make_weight(fmt, n, k, 511 + i)) for i, (n, k) in enumerate(((F, K), (F, K), (K, F), (K, K)))]
    x, g = make_x(1, K, 515), np.ones(K, np.float16)
    xb, gb, act, res, out = ctx.upload(x.view(np.uint16)), ctx.upload(g.view(np.uint16)), ctx.alloc(F * 2), ctx.alloc(K * 2), ctx.alloc(K * 2)

    def enqueue():
        ctx.rmsnorm_gate_up_silu(1, F, K, xb, gb, 1e-5, ws[0].buf, ws[1].buf, act)
        ctx.linear_add(1, K, F, act, ws[2].buf, res)
        ctx.rmsnorm_linear(1, K, K, res, gb, 1e-5, ws[3].buf, out)

    def read():
        ctx.sync()
        return [ctx.download(b, (n,), np.uint16) for b, n in ((act, F), (res, K), (out, K))]

    ctx.upload(x.view(np.uint16), res)
    enqueue()
    want = read()
    (Wg, sg), (Wu, su) = make_weight(fmt, F, K, 511), make_weight(fmt, F, K, 512)
    check_close(want[0].view(np.float16)[None], cpu.linear_swiglu(fmt, cpu.rmsnorm(x, g, 1e-5), Wg, sg, Wu, su), tol=2e-3, what=f"swiglu {fmt}")
    ctx.plan_begin()
    enqueue()
    plan = ctx.plan_end()
    assert ctx.L.nn_plan_num_resident_runs(plan) == 1
    for _ in range(2):
        ctx.upload(x.view(np.uint16), res)
        ctx.plan_launch(plan)
        for got, e in zip(read(), want):
            assert np.array_equal(got, e)
    ctx.L.nn_plan_free(plan)
    for w in ws:
        w.release()
    for b in (xb, gb, act, res, out):
        ctx.free(b)
