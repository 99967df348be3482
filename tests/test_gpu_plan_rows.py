"""Resident steps whose activation rows are the longest that stay in registers between fetch and staging, and the first longer
ones (3072 values with a norm, 6144 without), and rows of fewer pieces than threads: the bits of the separate launches."""
import importlib

import numpy as np
import pytest

from helpers import make_weight, make_x
from test_gpu_plan import _poison, _snapshot

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", ["int8", "fp16", "q4"])
@pytest.mark.parametrize("H,F", [(3072, 6144), (3136, 6208), (256, 320)])
def test_row_lengths(nnb, ctx, fmt, H, F):
    synth, dstep = importlib.import_module("adreno_llms_b200.synth"), importlib.import_module("adreno_llms_b200.decode_step")
    shape = synth.ModelShape("rows", H, 2, 256, 128, F, 512)
    step = dstep.DecodeStep(ctx, shape, fmt, M=1, n_sets=1, norm=True, chained=True)
    _poison(ctx, step)
    step.enqueue(0)
    ctx.sync()
    eager = _snapshot(ctx, step)
    assert np.isfinite(eager["logits"].view(np.float16).astype(np.float32)).all()
    step.record()
    assert step.resident_runs() >= 1
    for rep in range(2):
        step.reset_residual()
        _poison(ctx, step)
        step.launch(0)
        ctx.sync()
        now = _snapshot(ctx, step)
        for k, v in eager.items():
            assert np.array_equal(now[k], v), f"{fmt} {H}/{F} {k} replay {rep}"
    for st in step.sets:
        for w in st.values():
            w.release()


@pytest.mark.parametrize("fmt", ["fp16", "int8", "q4"])
def test_rows_of_other_lengths_and_norms_from_one_buffer(nnb, ctx, fmt):
    """Operators of a run that read the same buffer, but more of it or with another eps, stage it anew."""
    N = 4800   # (more tiles than blocks: every block has a part of every operator)
    x, g = make_x(1, 1024, 71), np.ones(1024, np.float16)
    xb, gb = ctx.upload(x.view(np.uint16)), ctx.upload(g.view(np.uint16))
    qs = {K: nnb.QuantWeight(ctx, fmt, *make_weight(fmt, N, K, 72 + K)) for K in (512, 1024)}
    calls = [lambda o: ctx.linear(1, N, 512, xb, qs[512].buf, o), lambda o: ctx.linear(1, N, 1024, xb, qs[1024].buf, o),
             lambda o: ctx.rmsnorm_linear(1, N, 1024, xb, gb, 1e-5, qs[1024].buf, o), lambda o: ctx.rmsnorm_linear(1, N, 1024, xb, gb, 3.0, qs[1024].buf, o),
             lambda o: ctx.rmsnorm_linear(1, N, 512, xb, gb, 3.0, qs[512].buf, o)]
    outs = [ctx.alloc(N * 2) for _ in calls]
    for f, o in zip(calls, outs):
        f(o)
    want = [ctx.download(o, (N,), np.uint16) for o in outs]
    for o in outs:
        ctx.upload(np.full(N, 0x7E00, np.uint16), o)
    ctx.plan_begin()
    for f, o in zip(calls, outs):
        f(o)
    plan = ctx.plan_end()
    assert ctx.L.nn_plan_num_resident_runs(plan) == 1
    ctx.plan_launch(plan)
    ctx.sync()
    for i, (o, w) in enumerate(zip(outs, want)):
        assert np.array_equal(ctx.download(o, (N,), np.uint16), w), i
    ctx.L.nn_plan_free(plan)
    for q in qs.values():
        q.release()
    for p in [xb, gb] + outs:
        ctx.free(p)
