"""Batches of 2..16 rows on both sides of the lines between the batch kernel and the streaming kernel: a row's bits are the single call's,
a recorded call's those of the eager one, and the launches say which of the two kernels ran (lines as for the 148 multiprocessors of a B200)."""
import numpy as np
import pytest

from helpers import alloc_with_canary, check_canary, make_weight, make_x

pytestmark = pytest.mark.gpu


# (Q4 9664 x 896: 302 tiles, so that some blocks take a second one)
@pytest.mark.parametrize("fmt,N,K", [("fp16", 321, 2752), ("int8", 321, 4864), ("q4", 130, 4608), ("q4", 9664, 896)])
def test_rows_of_several_groups_and_tiles(nnb, ctx, fmt, N, K):
    (W, s), (U, u) = make_weight(fmt, N, K, 401), make_weight(fmt, N, K, 402)
    qw, qu = nnb.QuantWeight(ctx, fmt, W, s), nnb.QuantWeight(ctx, fmt, U, u)
    x, r = make_x(16, K, 403), make_x(16, N, 404)
    xb, ob = ctx.upload(x.view(np.uint16)), alloc_with_canary(ctx, 16 * N * 2)
    calls = {
        "plain": lambda M, m: ctx.linear(M, N, K, xb + m * K * 2, qw.buf, ob + m * N * 2),
        "add": lambda M, m: ctx.linear_add(M, N, K, xb + m * K * 2, qw.buf, ob + m * N * 2),
        "swiglu": lambda M, m: ctx.fused_gate_up_silu(M, N, K, xb + m * K * 2, qw.buf, qu.buf, ob + m * N * 2),
    }
    for form, call in calls.items():
        def run(M, step):
            ctx.upload(r.view(np.uint16), ob)
            for m in range(0, M, step):
                call(min(step, M - m), m)
            return ctx.download(ob, (M, N), np.uint16)
        want = run(16, 1)
        for M in (2, 8, 9, 16):
            before = ctx.launch_count()
            got = run(M, 16)
            launches = ctx.launch_count() - before
            if (fmt, K, form, M) == ("q4", 4608, "swiglu", 16):
                assert launches == 2   # (no room beside two stages: the streaming kernel, in smaller chunks, so other sums)
                continue
            if fmt != "q4" or M * K >= 12288:   # (fewer values in Q4 are one launch in both kernels)
                assert launches == (2 if (fmt, N, M) == ("q4", 9664, 16) else 1), (form, M)
            assert np.array_equal(got, want[:M]), f"{fmt} {N}x{K} {form} M={M}"
    check_canary(ctx, ob, 16 * N * 2, f"{fmt} {N}x{K}")
    for q in (qw, qu):
        q.release()
    for p in (xb, ob):
        ctx.free(p)


@pytest.mark.parametrize("fmt,N,K,M,launches", [("int8", 9601, 384, 9, 1), ("int8", 10305, 384, 9, 2), ("int8", 5120, 384, 16, 1), ("int8", 5153, 384, 16, 2), ("int8", 9600, 576, 16, 1),
                                                ("int8", 9760, 576, 16, 2), ("int8", 4800, 2112, 2, 2), ("int8", 4800, 2048, 2, 1), ("q4", 500, 2624, 16, 2), ("q4", 500, 2048, 16, 1)])
def test_plain_rows_on_both_sides_of_a_line(nnb, ctx, fmt, N, K, M, launches):
    W, s = make_weight(fmt, N, K, 441)
    qw = nnb.QuantWeight(ctx, fmt, W, s)
    xb, ob = ctx.upload(make_x(M, K, 442).view(np.uint16)), alloc_with_canary(ctx, M * N * 2)
    for m in range(M):
        ctx.linear(1, N, K, xb + m * K * 2, qw.buf, ob + m * N * 2)
    want = ctx.download(ob, (M, N), np.uint16)
    ctx.upload(np.full((M, N), 0x7E00, np.uint16), ob)
    before = ctx.launch_count()
    ctx.linear(M, N, K, xb, qw.buf, ob)
    assert ctx.launch_count() - before == launches
    assert np.array_equal(ctx.download(ob, (M, N), np.uint16), want)
    check_canary(ctx, ob, M * N * 2, f"{fmt} {N}x{K}")
    qw.release()
    for p in (xb, ob):
        ctx.free(p)


@pytest.mark.parametrize("fmt", ["fp16", "int8", "q4"])
@pytest.mark.parametrize("N,K", [(70, 1088), (64, 4608), (64, 4672), (2048, 8192)])   # the longest row that up to 8 rows are normalised in the kernel with, and longer ones
def test_a_norm_gives_the_same_bits_recorded_and_row_by_row(nnb, ctx, fmt, N, K):
    W, s = make_weight(fmt, N, K, 411)
    qw = nnb.QuantWeight(ctx, fmt, W, s)
    x, g = make_x(16, K, 412), (1.0 + 0.1 * np.random.default_rng(413).standard_normal(K)).astype(np.float16)
    x[2] *= np.float16(30.0)
    xb, gb, ob = ctx.upload(x.view(np.uint16)), ctx.upload(g.view(np.uint16)), ctx.alloc(16 * N * 2)
    for m in range(16):
        ctx.rmsnorm_linear(1, N, K, xb + m * K * 2, gb, 1e-5, qw.buf, ob + m * N * 2)
    single = ctx.download(ob, (16, N), np.uint16)
    for M in (2, 8, 16):
        ctx.rmsnorm_linear(M, N, K, xb, gb, 1e-5, qw.buf, ob)
        want = ctx.download(ob, (M, N), np.uint16)
        if K <= 4672:   # (longer rows in Q4 may go to the streaming kernel in smaller chunks: other sums than the single call's)
            assert np.array_equal(want, single[:M]), f"{fmt} {N}x{K} M={M}"
        ctx.plan_begin()
        ctx.rmsnorm_linear(M, N, K, xb, gb, 1e-5, qw.buf, ob)
        plan = ctx.plan_end()
        ctx.upload(np.full((M, N), 0x7E00, np.uint16), ob)
        ctx.plan_launch(plan)
        assert np.array_equal(ctx.download(ob, (M, N), np.uint16), want), f"{fmt} {N}x{K} M={M} recorded"
        ctx.sync()
        ctx.L.nn_plan_free(plan)
    qw.release()
    for p in (xb, gb, ob):
        ctx.free(p)


# Gate and up with the norm, on both sides of the lines between the two kernels (on a B200: 148 multiprocessors); blocks that take several tiles
ONE_LAUNCH = {("q4", 8192, 16), ("q4", 4864, 2), ("q4", 2300, 2), ("q4", 2300, 8), ("int8", 4864, 16), ("int8", 2300, 2), ("int8", 2300, 8), ("int8", 2300, 9),
              ("int8", 2300, 16), ("fp16", 9400, 2), ("fp16", 9400, 8), ("fp16", 4864, 2), ("fp16", 4864, 8), ("fp16", 4864, 9),
              ("fp16", 4864, 16)}


@pytest.mark.parametrize("fmt,N,K", [("q4", 2300, 320), ("q4", 4864, 896), ("q4", 8192, 2752), ("int8", 4864, 896), ("int8", 2300, 320), ("fp16", 9400, 320), ("fp16", 4864, 896)])
def test_gate_and_up_with_the_norm(nnb, ctx, fmt, N, K):
    (W, s), (U, u) = make_weight(fmt, N, K, 421), make_weight(fmt, N, K, 422)
    qw, qu = nnb.QuantWeight(ctx, fmt, W, s), nnb.QuantWeight(ctx, fmt, U, u)
    x, g = make_x(16, K, 423), (1.0 + 0.1 * np.random.default_rng(424).standard_normal(K)).astype(np.float16)
    xb, gb, ob = ctx.upload(x.view(np.uint16)), ctx.upload(g.view(np.uint16)), alloc_with_canary(ctx, 16 * N * 2)
    for m in range(16):
        ctx.rmsnorm_gate_up_silu(1, N, K, xb + m * K * 2, gb, 1e-5, qw.buf, qu.buf, ob + m * N * 2)
    single = ctx.download(ob, (16, N), np.uint16)
    for M in (2, 8, 9, 16):
        ctx.upload(np.full((M, N), 0x7E00, np.uint16), ob)
        ctx.rmsnorm_gate_up_silu(M, N, K, xb, gb, 1e-5, qw.buf, qu.buf, ob)
        want = ctx.download(ob, (M, N), np.uint16)
        assert np.array_equal(want, single[:M]), f"{fmt} {N}x{K} M={M}"
        ctx.upload(np.full((M, N), 0x7E00, np.uint16), ob)
        ctx.plan_begin()
        ctx.rmsnorm_gate_up_silu(M, N, K, xb, gb, 1e-5, qw.buf, qu.buf, ob)
        plan = ctx.plan_end()
        ctx.plan_launch(plan)
        assert np.array_equal(ctx.download(ob, (M, N), np.uint16), want), f"{fmt} {N}x{K} M={M} recorded"
        # one launch where the norm is applied in the projection's
        assert ctx.L.nn_plan_num_recorded(plan) == (1 if (fmt, N, M) in ONE_LAUNCH else 2), (fmt, N, K, M)
        ctx.sync()
        ctx.L.nn_plan_free(plan)
    check_canary(ctx, ob, 16 * N * 2, f"{fmt} {N}x{K}")
    for q in (qw, qu):
        q.release()
    for p in (xb, gb, ob):
        ctx.free(p)


@pytest.mark.parametrize("fmt", ["fp16", "int8", "q4"])
@pytest.mark.parametrize("K", [576, 1024])
def test_outputs_over_the_rows(nnb, ctx, fmt, K):
    """A call of 2..16 rows has read its rows before it writes over them (the staging launch copies them)."""
    (W, s), (U, u) = make_weight(fmt, K, K, 431), make_weight(fmt, K, K, 432)
    qw, qu = nnb.QuantWeight(ctx, fmt, W, s), nnb.QuantWeight(ctx, fmt, U, u)
    x, g = make_x(16, K, 433), (1.0 + 0.1 * np.random.default_rng(434).standard_normal(K)).astype(np.float16)
    xb, gb, ob = ctx.upload(x.view(np.uint16)), ctx.upload(g.view(np.uint16)), ctx.alloc(16 * K * 2)
    calls = {
        "plain": lambda M, out: ctx.linear(M, K, K, xb, qw.buf, out),
        "add": lambda M, out: ctx.linear_add(M, K, K, xb, qw.buf, out),
        "swiglu": lambda M, out: ctx.fused_gate_up_silu(M, K, K, xb, qw.buf, qu.buf, out),
        "norm": lambda M, out: ctx.rmsnorm_linear(M, K, K, xb, gb, 1e-5, qw.buf, out),
    }
    for form, call in calls.items():
        for M in (2, 8, 16):
            ctx.upload(x.view(np.uint16), xb)
            ctx.upload(x.view(np.uint16), ob)
            call(M, ob)
            want = ctx.download(ob, (M, K), np.uint16)
            for recorded in (False, True):
                ctx.upload(x.view(np.uint16), xb)
                before = ctx.launch_count()
                if recorded:
                    ctx.plan_begin()
                    call(M, xb)
                    plan = ctx.plan_end()
                    assert ctx.L.nn_plan_num_recorded(plan) == 2, (form, M)
                    ctx.plan_launch(plan)
                else:
                    call(M, xb)
                    assert ctx.launch_count() - before == 2, (form, M)
                assert np.array_equal(ctx.download(xb, (M, K), np.uint16), want), f"{fmt} {form} M={M} recorded={recorded}"
                ctx.sync()
                if recorded:
                    ctx.L.nn_plan_free(plan)
    for q in (qw, qu):
        q.release()
    for p in (xb, gb, ob):
        ctx.free(p)
