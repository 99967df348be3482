"""2..16 rows of an operator whose tiles split K, in one launch: every row carries the bits of the single call, at the edges of tiles,
stages, columns and rows, for each way the kernel finishes a tile; a norm inside a recorded launch gives the bits of the staged one."""
import numpy as np
import pytest

from helpers import alloc_with_canary, check_canary, make_weight, make_x

pytestmark = pytest.mark.gpu

# (N, K): odd and even row counts around the tile (16, 32), rows of one stage and of several, whole and part 128-byte columns, few tiles and
# more than blocks at a time
CASES = [("fp16", 31, 128), ("fp16", 129, 1088), ("fp16", 2050, 320), ("int8", 17, 256), ("int8", 576, 576), ("int8", 321, 4864), ("int8", 9601, 448),
         ("q4", 33, 512), ("q4", 576, 896), ("q4", 130, 4608), ("q4", 9700, 256)]


@pytest.mark.parametrize("fmt,N,K", CASES)
def test_rows_are_the_single_calls(nnb, ctx, fmt, N, K):
    (W, s), (U, u) = make_weight(fmt, N, K, 401), make_weight(fmt, N, K, 402)
    qw, qu = nnb.QuantWeight(ctx, fmt, W, s), nnb.QuantWeight(ctx, fmt, U, u)
    x, r = make_x(16, K, 403), make_x(16, N, 404)
    x[1] *= np.float16(20.0)
    b = [make_x(1, n, 405)[0] for n in (N, 5, 40)]
    (V, v), (Z, z) = make_weight(fmt, 5, K, 406), make_weight(fmt, 40, K, 407)
    qv, qz = nnb.QuantWeight(ctx, fmt, V, v), nnb.QuantWeight(ctx, fmt, Z, z)
    xb, ob, k, w = ctx.upload(x.view(np.uint16)), alloc_with_canary(ctx, 16 * N * 2), ctx.alloc(16 * 5 * 2), ctx.alloc(16 * 40 * 2)
    bb = [ctx.upload(t.view(np.uint16)) for t in b]
    row = lambda p, m, n: p + m * n * 2  # noqa: E731
    calls = {
        "plain": lambda M, m: ctx.linear(M, N, K, row(xb, m, K), qw.buf, row(ob, m, N)),
        "add": lambda M, m: ctx.linear_add(M, N, K, row(xb, m, K), qw.buf, row(ob, m, N)),
        "gate": lambda M, m: ctx.linear_silu_gate_fused(M, N, K, row(xb, m, K), qw.buf, row(ob, m, N)),
        "swiglu": lambda M, m: ctx.fused_gate_up_silu(M, N, K, row(xb, m, K), qw.buf, qu.buf, row(ob, m, N)),
        "qkv": lambda M, m: ctx.linear_qkv_bias(M, K, row(xb, m, K), qw.buf, N, qv.buf, 5, qz.buf, 40, *bb, row(ob, m, N), row(k, m, 5), row(w, m, 40)),
    }
    for form, call in calls.items():
        def run(M, step):
            ctx.upload(r.view(np.uint16), ob)
            for buf, n in ((k, 5), (w, 40)):
                ctx.upload(np.full((16, n), 0x7E00, np.uint16), buf)
            for m in range(0, M, step):
                call(min(step, M - m), m)
            return [ctx.download(buf, (16, n), np.uint16)[:M] for buf, n in ((ob, N), (k, 5), (w, 40))]
        want = run(16, 1)
        for M in (2, 3, 8) if fmt == "q4" and K > 1088 else (2, 3, 8, 9, 16):   # (16 long Q4 rows: the streaming kernel, in smaller chunks)
            before = ctx.launch_count()
            got = run(M, 16)
            assert ctx.launch_count() - before == 1 or K > 1088 or (fmt, form) == ("q4", "swiglu") and M > 8, (form, M)
            for g, e in zip(got, want):
                assert np.array_equal(g, e[:M]), f"{fmt} {N}x{K} {form} M={M}"
    check_canary(ctx, ob, 16 * N * 2, f"{fmt} {N}x{K}")
    for q in (qw, qu, qv, qz):
        q.release()
    for p in [xb, ob, k, w] + bb:
        ctx.free(p)


@pytest.mark.parametrize("fmt", ["fp16", "int8", "q4"])
@pytest.mark.parametrize("N,K", [(96, 256), (70, 1024), (70, 1088), (64, 4608), (64, 4672)])   # passes of 1024 values; the longest row, and one more
def test_norm_in_a_recorded_launch(nnb, ctx, fmt, N, K):
    W, s = make_weight(fmt, N, K, 411)
    qw = nnb.QuantWeight(ctx, fmt, W, s)
    x, g = make_x(16, K, 412), (1.0 + 0.1 * np.random.default_rng(413).standard_normal(K)).astype(np.float16)
    x[2] *= np.float16(30.0)
    xb, gb, ob = ctx.upload(x.view(np.uint16)), ctx.upload(g.view(np.uint16)), ctx.alloc(16 * N * 2)
    for M in (2, 5, 8, 11, 16):
        ctx.rmsnorm_linear(M, N, K, xb, gb, 1e-5, qw.buf, ob)
        want = ctx.download(ob, (M, N), np.uint16)
        ctx.plan_begin()
        ctx.rmsnorm_linear(M, N, K, xb, gb, 1e-5, qw.buf, ob)
        plan = ctx.plan_end()
        for _ in range(2):
            ctx.upload(np.full((M, N), 0x7E00, np.uint16), ob)
            ctx.plan_launch(plan)
            assert np.array_equal(ctx.download(ob, (M, N), np.uint16), want), f"{fmt} {N}x{K} M={M}"
        ctx.sync()
        ctx.L.nn_plan_free(plan)
    qw.release()
    for p in (xb, gb, ob):
        ctx.free(p)
