"""Resident steps whose activation rows are the longest that stay in registers between fetch and staging, and the first longer
ones (3072 values with a norm, 6144 without), and rows of fewer pieces than threads: the bits of the separate launches."""
import importlib

import numpy as np
import pytest

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
