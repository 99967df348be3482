"""The work a host program has this library do, as timed cases.

Three kinds of case, over the library's whole range:

  linear    one projection called on its own: the smallest a decode loop issues, the large lm_head and
            FFN matrices, batched decode rows and prefill rows (options: plain, gate/up/SiLU over two
            weights, q/k/v with bias, lm_head with the greedy pick)
  step      a decode step of a whole model for 1..16 sequences, recorded once and replayed per token,
            with the model's data flow: every projection waits for the one before it, the layer norms
            ride in the projections, each layer's k and v go to buffers of their own (the cache rows)
  prefill   a prompt of M tokens through the same layers, called operator by operator (prompt lengths
            vary, so nothing is recorded), then the logits and the greedy token of its last row

Attention itself is not on the library's path; q stands in for its output, as in the decode step of
adreno-llms_b200/decode_step.py.  Weights are N(0, 0.02) quantised to the three stored formats,
activations N(0, 1).
"""
import importlib.util
import math
import os
import sys

import torch

FORMATS = ("fp16", "int8", "q4")
EPS = 1e-5

# hidden, layers, kv_dim, ffn, vocab, q/k/v bias: the three model shapes this repository is configured for
SMOLLM2_135M = dict(hidden=576, layers=30, kv_dim=192, ffn=1536, vocab=49152, bias=False)
QWEN25_05B = dict(hidden=896, layers=24, kv_dim=128, ffn=4864, vocab=151936, bias=True)
LFM25_350M = dict(hidden=1024, layers=16, kv_dim=512, ffn=4608, vocab=65536, bias=False)


def listed():
    return [
        # the smallest call: one per-layer projection of the 135M shape, a few microseconds of latency
        dict(name="gemv_int8_1536x576", kind="linear", op="linear", fmt="int8", M=1, N=1536, K=576),
        # the tied lm_head of the largest vocabulary with its greedy pick, one token
        dict(name="lm_head_int8_pick", kind="linear", op="argmax", fmt="int8", M=1, N=151936, K=896),
        # a scaled-up 4-bit FFN matrix: one token, and a batch of 32 sequences
        dict(name="ffn_q4_m1", kind="linear", op="linear", fmt="q4", M=1, N=28672, K=8192),
        dict(name="ffn_q4_m32", kind="linear", op="linear", fmt="q4", M=32, N=28672, K=8192),
        # logits of 256 rows at once (scoring, speculative decoding), and of a whole long prompt
        dict(name="lm_head_int8_m256", kind="linear", op="linear", fmt="int8", M=256, N=151936, K=896),
        dict(name="lm_head_fp16_m2048", kind="linear", op="linear", fmt="fp16", M=2048, N=151936, K=896),
        # a token of one user: the smallest model int8, the largest fp16
        dict(name="step_135m_int8_m1", kind="step", fmt="int8", M=1, **SMOLLM2_135M),
        dict(name="step_500m_fp16_m1", kind="step", fmt="fp16", M=1, **QWEN25_05B),
        # a token of each of several users
        dict(name="step_350m_q4_m8", kind="step", fmt="q4", M=8, **LFM25_350M),
        dict(name="step_500m_int8_m16", kind="step", fmt="int8", M=16, **QWEN25_05B),
        # prompts: a long one, and a short one of an odd length
        dict(name="prefill_500m_fp16_512", kind="prefill", fmt="fp16", M=512, **QWEN25_05B),
        dict(name="prefill_350m_q4_77", kind="prefill", fmt="q4", M=77, **LFM25_350M),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


MOST_FLOPS = 2.0 * 2048 * 151936 * 896   # the largest listed case
MOST_WEIGHTS = 28672 * 8192              # of one operator
MOST_PARAMS = 5.0e8                      # of one model


def _layer_params(c):
    return c["hidden"] * (2 * c["hidden"] + 2 * c["kv_dim"] + 3 * c["ffn"])


def draw(rng):
    kind = rng.choice(("linear", "linear", "step", "step", "prefill"))
    fmt = rng.choice(FORMATS)
    if kind == "linear":
        M = int(_log_uniform(rng, 1, 17)) if rng.random() < 0.5 else int(_log_uniform(rng, 17, 2049))
        op = rng.choice(("linear", "linear", "gate_up", "qkv", "argmax"))
        if op == "argmax":
            M = 1
        K = 32 * round(_log_uniform(rng, 256, 8192) / 32)
        N = int(_log_uniform(rng, 8192, 152000) if op == "argmax" else _log_uniform(rng, 256, 32768))
        N = max(64, min(N, MOST_WEIGHTS // K // (2 if op == "gate_up" else 1)))
        return dict(kind=kind, op=op, fmt=fmt, M=M, N=N, K=K)
    hidden = 64 * int(_log_uniform(rng, 4, 25))
    c = dict(kind=kind, fmt=fmt, M=1, hidden=hidden, layers=rng.randint(4, 30), kv_dim=64 * rng.randint(1, max(1, hidden // 128)),
             ffn=64 * round(hidden * rng.uniform(2.5, 5.5) / 64), vocab=int(_log_uniform(rng, 8192, 152000)), bias=rng.random() < 0.5)
    while c["layers"] * _layer_params(c) + c["vocab"] * hidden > MOST_PARAMS:
        c["layers"] -= 1
    if kind == "step":
        c["M"] = int(_log_uniform(rng, 1, 17))
    else:
        c["M"] = max(17, min(int(_log_uniform(rng, 17, 2049)), int(0.9 * MOST_FLOPS / (2.0 * c["layers"] * _layer_params(c)))))
    return c


# ---- what one pass cannot do without ------------------------------------------------------------
def _weight_bytes(fmt, n, k):
    return 2 * n * k if fmt == "fp16" else n * k + 2 * n if fmt == "int8" else n * k // 2 + 2 * n * (k // 32)


def _qkv_rows(n):
    """q, k and v rows of an N-row q/k/v projection: four query heads to one of k and v."""
    kv = max(1, n // 6)
    return n - 2 * kv, kv


def work(case):
    c, fmt, M = case, case["fmt"], case["M"]
    if c["kind"] == "linear":
        nw = 2 if c["op"] == "gate_up" else 1
        b = nw * _weight_bytes(fmt, c["N"], c["K"]) + 2 * M * (c["K"] + c["N"])
        if c["op"] == "qkv":
            b += 2 * c["N"]
        if c["op"] == "argmax":
            b += 4
        return {"bytes": b, "flops": 2.0 * nw * M * c["N"] * c["K"]}
    H, F, KV, V, L = c["hidden"], c["ffn"], c["kv_dim"], c["vocab"], c["layers"]
    layer = _weight_bytes(fmt, 2 * H, H) + 2 * _weight_bytes(fmt, KV, H) + 2 * _weight_bytes(fmt, F, H) + _weight_bytes(fmt, H, F)
    layer += 2 * 2 * H + (2 * (H + 2 * KV) if c["bias"] else 0)          # norm weights, biases
    layer += 2 * 2 * M * KV                                              # k and v rows written
    rows = M if c["kind"] == "step" else 1                               # rows whose logits are wanted
    b = L * layer + _weight_bytes(fmt, V, H) + 2 * H + 2 * 2 * M * H + 2 * rows * V + (4 if rows == 1 else 0)
    return {"bytes": b, "flops": 2.0 * M * L * _layer_params(c) + 2.0 * rows * V * H}


def tolerance(case):
    # fp16 results of fp32 sums: half a unit in the last place is 2.4e-4 of a value, and where activations or
    # 4-bit weights are rounded to fp16 on the way the sums differ by as much again; a whole model compounds
    # that over its layers.
    return {"rel": 1e-3} if case["kind"] == "linear" else {"rel": 6e-3}


# ---- the library ---------------------------------------------------------------------------------
def _package():
    name = "adreno_llms_b200"
    if name not in sys.modules:
        path = os.path.join(os.getcwd(), "adreno-llms_b200", "__init__.py")
        spec = importlib.util.spec_from_file_location(name, path, submodule_search_locations=[os.path.dirname(path)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


_context = None


def _ctx():
    """The process's one context, as a serving program keeps it."""
    global _context
    if _context is None:
        torch.cuda.init()
        _context = _package().Context(torch.cuda.current_device())
    return _context


class _Inputs:
    """Seeded device tensors, and weights registered with the library for as long as this object lives."""

    def __init__(self, ctx, fmt, seed):
        self.ctx, self.fmt = ctx, fmt
        self.gen = torch.Generator(device="cuda")
        self.gen.manual_seed(seed)
        self.kept, self.registered, self.pending, self.plan = [], [], [], None

    def half(self, *shape, std=1.0, mean=0.0):
        t = torch.randn(shape, generator=self.gen, device="cuda", dtype=torch.float16).mul_(std)
        if mean:
            t.add_(mean)
        self.kept.append(t)
        return t

    def empty(self, *shape, dtype=torch.float16):
        t = torch.zeros(shape, device="cuda", dtype=dtype)
        self.kept.append(t)
        return t

    def weight(self, n, k):
        """One weight in its stored layout; returns its device pointer."""
        w = torch.randn((n, k), generator=self.gen, device="cuda", dtype=torch.float16).mul_(0.02)
        if self.fmt == "fp16":
            self.kept.append(w)
            return w.data_ptr()
        if self.fmt == "int8":
            codes, scale = torch.empty((n, k), device="cuda", dtype=torch.int8), torch.empty((n,), device="cuda", dtype=torch.float16)
        else:
            codes, scale = torch.empty((n, k // 2), device="cuda", dtype=torch.uint8), torch.empty((n, k // 32), device="cuda", dtype=torch.float16)
        rows = max(1, (1 << 25) // k)
        for r in range(0, n, rows):
            x = w[r:r + rows].float()
            if self.fmt == "int8":
                s = x.abs().amax(dim=1).div_(127.0)
                s = torch.where(s > 0, s, torch.ones_like(s))
                codes[r:r + rows] = torch.round(x / s[:, None]).clamp_(-127, 127).to(torch.int8)
                scale[r:r + rows] = s.half()
            else:
                x = x.view(x.shape[0], k // 32, 32)
                s = x.abs().amax(dim=2).div_(7.0)
                s = torch.where(s > 0, s, torch.ones_like(s))
                q = (torch.round(x / s[:, :, None]).clamp_(-7, 7) + 8).to(torch.uint8).view(x.shape[0], k)
                codes[r:r + rows] = q[:, 0::2] | (q[:, 1::2] << 4)
                scale[r:r + rows] = s.half()
        self.kept += [codes, scale]
        self.pending.append((codes.data_ptr(), scale.data_ptr(), n, k))
        return codes.data_ptr()

    def register(self):
        """Registration reads the scales on the library's stream: the tensors must be there."""
        torch.cuda.synchronize()
        for w, s, n, k in self.pending:
            (self.ctx.register_int8 if self.fmt == "int8" else self.ctx.register_q4)(w, s, n, k)
            self.registered.append(w)
        self.pending = []
        self.ctx.sync()

    def __del__(self):
        L, h = self.ctx.L, self.ctx.h
        if h:
            L.nn_sync(h)
            if self.plan:
                L.nn_plan_free(self.plan)
            for w in self.registered:
                L.nn_unregister_weight(h, w)


def _copy(ctx, dst, src):
    rc = ctx.L.nn_buf_copy(ctx.h, dst.data_ptr(), src.data_ptr(), src.numel() * src.element_size())
    if rc:
        raise RuntimeError("nn_buf_copy failed")


# ---- one projection --------------------------------------------------------------------------------
def _prepare_linear(ctx, c, seed):
    s = _Inputs(ctx, c["fmt"], seed)
    M, N, K, op = c["M"], c["N"], c["K"], c["op"]
    x = s.half(M, K)
    if op == "gate_up":
        wg, wu, out = s.weight(N, K), s.weight(N, K), s.empty(M, N)
        call, outs = (ctx.fused_gate_up_silu, (M, N, K, x.data_ptr(), wg, wu, out.data_ptr())), [out]
    elif op == "qkv":
        nq, nkv = _qkv_rows(N)
        w = [s.weight(n, K) for n in (nq, nkv, nkv)]
        b = [s.half(n, std=0.5) for n in (nq, nkv, nkv)]
        outs = [s.empty(M, n) for n in (nq, nkv, nkv)]
        call = (ctx.linear_qkv_bias, (M, K, x.data_ptr(), w[0], nq, w[1], nkv, w[2], nkv, *[t.data_ptr() for t in b], *[t.data_ptr() for t in outs]))
    elif op == "argmax":
        w, logits, token = s.weight(N, K), s.empty(N), s.empty(1, dtype=torch.int32)
        call, outs = (ctx.linear_argmax, (N, K, x.data_ptr(), w, logits.data_ptr(), token.data_ptr())), [logits, token]
    else:
        w, out = s.weight(N, K), s.empty(M, N)
        call, outs = (ctx.linear, (M, N, K, x.data_ptr(), w, out.data_ptr())), [out]
    s.register()
    s.calls, s.outs = [call], outs
    return s


# ---- a whole model ---------------------------------------------------------------------------------
def _prepare_model(ctx, c, seed):
    s = _Inputs(ctx, c["fmt"], seed)
    M, H, F, KV, V, L = c["M"], c["hidden"], c["ffn"], c["kv_dim"], c["vocab"], c["layers"]
    hidden, resid = s.half(M, H), s.empty(M, H)          # the embedded tokens, and the residual stream
    q, act = s.empty(M, H), s.empty(M, F)
    k, v = s.empty(L, M, KV), s.empty(L, M, KV)
    rows = M if c["kind"] == "step" else 1
    logits = s.empty(rows, V)
    p = lambda t: t.data_ptr()  # noqa: E731
    calls = [(_copy, (ctx, resid, hidden))]
    for i in range(L):
        g1, g2 = s.half(H, std=0.1, mean=1.0), s.half(H, std=0.1, mean=1.0)
        wq, wk, wv, wo = s.weight(H, H), s.weight(KV, H), s.weight(KV, H), s.weight(H, H)
        wg, wu, wd = s.weight(F, H), s.weight(F, H), s.weight(H, F)
        if c["bias"]:
            b = [s.half(n, std=0.5) for n in (H, KV, KV)]
            calls.append((ctx.rmsnorm_linear_qkv_bias, (M, H, p(resid), p(g1), EPS, wq, H, wk, KV, wv, KV, *map(p, b), p(q), p(k[i]), p(v[i]))))
        else:
            calls.append((ctx.rmsnorm_linear_qkv, (M, H, p(resid), p(g1), EPS, wq, H, wk, KV, wv, KV, p(q), p(k[i]), p(v[i]))))
        calls.append((ctx.linear_add, (M, H, H, p(q), wo, p(resid))))
        calls.append((ctx.rmsnorm_gate_up_silu, (M, F, H, p(resid), p(g2), EPS, wg, wu, p(act))))
        calls.append((ctx.linear_add, (M, H, F, p(act), wd, p(resid))))
    g = s.half(H, std=0.1, mean=1.0)
    head = s.weight(V, H)
    calls.append((ctx.rmsnorm_linear, (rows, V, H, p(resid) + (M - rows) * H * 2, p(g), EPS, head, p(logits))))
    s.outs = {"hidden": resid, "k": k, "v": v, "logits": logits}
    if rows == 1:
        token = s.empty(1, dtype=torch.int32)
        calls.append((ctx.argmax, (V, p(logits), p(token))))
        s.outs["token"] = token
    s.register()
    s.calls = calls
    if c["kind"] == "step":
        ctx.plan_begin()
        for f, args in calls:
            f(*args)
        s.plan = ctx.plan_end()
        s.calls = [(ctx.plan_launch, (s.plan,))]
    return s


def prepare(case, seed):
    ctx = _ctx()
    return _prepare_linear(ctx, case, seed) if case["kind"] == "linear" else _prepare_model(ctx, case, seed)


def run(state):
    for f, args in state.calls:
        f(*args)
    return state.outs
