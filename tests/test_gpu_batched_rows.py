"""Batches whose staged activations do not fit in shared memory and travel with the weights, and the row-pair finish at odd row
counts: every row carries the bits of the single-token call, whichever way it was computed."""
import numpy as np
import pytest

from helpers import alloc_with_canary, check_canary, check_close, make_weight, make_x
from oracle import cpu

pytestmark = pytest.mark.gpu

# (N, K): tiles that split K and whole-row tiles, odd row counts, K of whole and of part stages
CASES = [("int8", 96, 4864), ("int8", 801, 5120), ("int8", 40001, 5184), ("fp16", 321, 8192), ("fp16", 40000, 7200), ("int8", 64, 16384),
         ("q4", 333, 1024), ("fp16", 77, 512), ("int8", 131, 640)]


@pytest.mark.parametrize("fmt,N,K", CASES)
def test_rows_of_a_batch_are_the_single_calls(nnb, ctx, fmt, N, K):
    W, s = make_weight(fmt, min(N, 1000), K, 301)
    rep = -(-N // W.shape[0])
    W = np.tile(W, (rep, 1))[:N]
    s = None if s is None else np.tile(s, (rep, 1) if s.ndim == 2 else rep)[:N]
    qw = nnb.QuantWeight(ctx, fmt, W, s)
    x, r = make_x(16, K, 302), make_x(16, N, 303)
    x[5] *= np.float16(0.05)
    xb, ob, rb = ctx.upload(x.view(np.uint16)), alloc_with_canary(ctx, 16 * N * 2), ctx.upload(r.view(np.uint16))
    plain, added = [], []
    for m in range(16):
        ctx.linear(1, N, K, xb + m * K * 2, qw.buf, ob)
        plain.append(ctx.download(ob, (N,), np.uint16))
        ctx.linear_add(1, N, K, xb + m * K * 2, qw.buf, rb + m * N * 2)
    added = ctx.download(rb, (16, N), np.uint16)
    for M in (2, 7, 9, 16):
        ctx.upload(np.full((M, N), 0x7E00, np.uint16), ob)
        ctx.linear(M, N, K, xb, qw.buf, ob)
        assert np.array_equal(ctx.download(ob, (M, N), np.uint16), np.stack(plain[:M])), f"{fmt} {N}x{K} M={M}"
        ctx.upload(r.view(np.uint16), ob)
        ctx.linear_add(M, N, K, xb, qw.buf, ob)
        assert np.array_equal(ctx.download(ob, (M, N), np.uint16), added[:M]), f"{fmt} {N}x{K} M={M} in place"
        check_canary(ctx, ob, 16 * N * 2, f"{fmt} {N}x{K} M={M}")
    qw.release()
    for b in (xb, ob, rb):
        ctx.free(b)


@pytest.mark.parametrize("M", [4, 9])
def test_balanced_launch_with_split_k(nnb, ctx, M):
    """Q4, long rows, 500 tiles of 32 rows dealt out as pipeline items: warp 0 adds the K parts of a tile and finishes it."""
    N, K = 16000, 8192
    W, s = make_weight("q4", 1000, K, 311)
    qw = nnb.QuantWeight(ctx, "q4", np.tile(W, (16, 1)), np.tile(s, (16, 1)))
    x, r = make_x(M, K, 312), make_x(M, N, 313)
    xb, ob = ctx.upload(x.view(np.uint16)), alloc_with_canary(ctx, M * N * 2)
    want = np.tile(x.astype(np.float64) @ cpu.dequant("q4", W, s).astype(np.float64).T, (1, 16))
    seen = None
    for rep in range(6):
        ctx.upload(r.view(np.uint16), ob)
        ctx.linear_add(M, N, K, xb, qw.buf, ob)
        got = ctx.download(ob, (M, N), np.uint16)
        check_close(got.view(np.float16), r.astype(np.float64) + want, what=f"q4 {N}x{K} M={M}")
        assert seen is None or np.array_equal(got, seen)
        seen = got
    check_canary(ctx, ob, M * N * 2, f"q4 {N}x{K} M={M}")
    qw.release()
    for b in (xb, ob):
        ctx.free(b)
