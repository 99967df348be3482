"""int8 sums are exact until a K quarter of a tile ends: terms that cancel leave nothing behind, whichever kernel takes the call."""
import numpy as np
import pytest

from helpers import alloc_with_canary, check_canary

pytestmark = pytest.mark.gpu


def _operands(N, K, seed):
    """Rows whose units of 64 values each hold 2^15 and -2^15 against equal codes, and small multiples of 2^-6 otherwise."""
    rng = np.random.default_rng(seed)
    W = rng.integers(-127, 128, (N, K)).astype(np.int8)
    x = (rng.integers(-64, 65, (16, K)) / 64.0).astype(np.float16)
    for u in range(0, K - 63, 64):
        W[:, u + 40] = W[:, u + 5]
        x[:, u + 5] = 32768.0
        x[:, u + 40] = -32768.0
    return W, x


def _bound(W, x):
    """Largest error of the sums: the fp32 roundings where a quarter's limb sums become one number (24-bit fixed point: the row's largest
    value is 2^15, so the last place is 2^-7 and every value here is held exactly), of the additions of the quarters and by the scale."""
    K = W.shape[1]
    chunk = (-(-K // 4) + 127) // 128 * 128
    if chunk > 384:
        chunk = 256
    fix, W = np.rint(x.astype(np.float64) * 128).astype(np.int64), W.astype(np.int64)
    limbs = (fix >> 16, (fix >> 8) & 255, fix & 255)
    quarters = [np.concatenate([np.arange(c, min(c + chunk, K)) for c in range(q * chunk, K, 4 * chunk)] or [np.zeros(0, np.int64)]) for q in range(4)]
    err = np.zeros((x.shape[0], W.shape[0]))
    total = np.zeros_like(err)
    for k in quarters:
        hi, mid, lo = (l[:, k] @ W[:, k].T for l in limbs)
        inner = mid * 256 + lo
        s = (hi * 65536 + inner) / 128.0
        err += 2.0 ** -24 * (np.abs(inner) + np.abs(mid) * 256 + np.abs(lo)) / 128.0 + 2.0 ** -24 * np.abs(s)
        total += np.abs(s)
    return err + 5 * 2.0 ** -24 * total


@pytest.mark.parametrize("N,K", [(40, 576), (577, 896), (64, 4864), (300, 1024)])
def test_cancelling_terms(nnb, ctx, N, K):
    W, x = _operands(N, K, 601)
    s = np.full(N, 2.0 ** -6, np.float16)
    qw = nnb.QuantWeight(ctx, "int8", W, s)
    want = (x.astype(np.float64) @ W.astype(np.float64).T) / 64
    bound = _bound(W, x) / 64
    xb, ob = ctx.upload(x.view(np.uint16)), alloc_with_canary(ctx, 16 * N * 2)

    def check(M, what):
        got = ctx.download(ob, (M, N), np.uint16).view(np.float16).astype(np.float64)
        rounding = np.spacing(np.abs(want[:M]).astype(np.float16)).astype(np.float64) / 2
        err = np.abs(got - want[:M])
        assert (err <= rounding + bound[:M]).all(), f"int8 {N}x{K} M={M} {what}: off by {(err - rounding - bound[:M]).max()}"

    for M in (1, 2, 8, 9, 16):
        ctx.linear(M, N, K, xb, qw.buf, ob)
        check(M, "called")
        # two operators of one token make a run of the resident kernel
        ctx.plan_begin()
        for _ in range(2):
            ctx.linear(M, N, K, xb, qw.buf, ob)
        plan = ctx.plan_end()
        ctx.upload(np.full((M, N), 0x7E00, np.uint16), ob)
        ctx.plan_launch(plan)
        ctx.sync()
        assert M > 1 or ctx.L.nn_plan_num_resident_runs(plan) == 1
        check(M, "recorded")
        ctx.L.nn_plan_free(plan)
    check_canary(ctx, ob, 16 * N * 2, f"int8 {N}x{K}")
    qw.release()
    for b in (xb, ob):
        ctx.free(b)


@pytest.mark.parametrize("M,N,K", [(1, 333, 896), (4, 333, 896), (11, 333, 896), (1, 333, 736), (3, 40000, 352), (16, 333, 736)])
def test_a_row_with_an_infinity(nnb, ctx, M, N, K):
    """A row that holds an Inf or a NaN gives NaN in all of its outputs, and no other row notices (736, 352: an odd number of 32 values)."""
    rng = np.random.default_rng(611)
    W, s = rng.integers(-127, 128, (N, K)).astype(np.int8), np.full(N, 2.0 ** -6, np.float16)
    qw = nnb.QuantWeight(ctx, "int8", W, s)
    x = rng.standard_normal((M, K)).astype(np.float16)
    xb, ob = ctx.upload(x.view(np.uint16)), ctx.alloc(M * N * 2)
    ctx.linear(M, N, K, xb, qw.buf, ob)
    want = ctx.download(ob, (M, N), np.uint16)
    for bad in (np.inf, np.nan):
        y = x.copy()
        y[M // 2, 77] = bad
        ctx.upload(y.view(np.uint16), xb)
        ctx.linear(M, N, K, xb, qw.buf, ob)
        got = ctx.download(ob, (M, N), np.uint16)
        assert np.isnan(got.view(np.float16)[M // 2]).all()
        others = [m for m in range(M) if m != M // 2]
        assert np.array_equal(got[others], want[others])
    qw.release()
    for b in (xb, ob):
        ctx.free(b)
