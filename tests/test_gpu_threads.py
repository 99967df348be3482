"""What the library keeps per thread goes with the thread."""
import threading

import numpy as np
import pytest

from helpers import make_weight, make_x

pytestmark = pytest.mark.gpu


def _resident_bytes():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * 4096


def test_threads_leave_no_memory_behind(nnb, ctx):
    N, K = 256, 512
    W, _ = make_weight("fp16", N, K, 1)
    q = nnb.QuantWeight(ctx, "fp16", W, None)
    xb, ob = ctx.upload(make_x(40, K, 2).view(np.uint16)), ctx.alloc(40 * N * 2)
    errors = []

    def work():
        try:
            own = ctx.alloc(40 * N * 2)              # (makes the device current in this thread)
            ctx.linear(40, N, K, xb, q.buf, own)     # the GEMM's tilings and tensor maps
            ctx.linear(1, N, K, xb, q.buf, own)      # the streaming kernel's tensor maps
            ctx.sync()
            ctx.free(own)
        except Exception as e:                       # noqa: BLE001
            errors.append(e)

    def run(n):
        for _ in range(n):
            t = threading.Thread(target=work)
            t.start()
            t.join()

    run(16)
    before = _resident_bytes()
    run(96)
    grown = _resident_bytes() - before
    assert not errors
    # a thread's tensor maps and tilings are some 500 KB
    assert grown < 16 * 500_000, f"{grown} bytes more after 96 threads"
    q.release()
    for b in (xb, ob):
        ctx.free(b)


@pytest.mark.parametrize("fmt", ["fp16", "int8", "q4"])
@pytest.mark.parametrize("M", [1, 2, 16, 40])
def test_a_projection_as_a_threads_first_call(nnb, ctx, fmt, M):
    N, K = 320, 768
    q = nnb.QuantWeight(ctx, fmt, *make_weight(fmt, N, K, 3))
    xb, ob = ctx.upload(make_x(M, K, 4).view(np.uint16)), ctx.alloc(M * N * 2)
    ctx.linear(M, N, K, xb, q.buf, ob)
    want = ctx.download(ob, (M, N), np.uint16)
    ctx.upload(np.full((M, N), 0x7E00, np.uint16), ob)
    ctx.sync()
    errors = []

    def work():
        try:
            ctx.linear(M, N, K, xb, q.buf, ob)
        except Exception as e:                       # noqa: BLE001
            errors.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not errors, errors
    assert np.array_equal(ctx.download(ob, (M, N), np.uint16), want)
    q.release()
    for b in (xb, ob):
        ctx.free(b)
