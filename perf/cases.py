"""The work that users of this library have it do, as cases that can be timed: MoE layers in decode
and in prefill, dense GEMVs, the head, dense GEMMs.

Weights are seeded random ggml blocks with the distributions of the package's synthetic tensors
(every byte pattern is a valid block; the f16 block scales come from a small positive range), made
on the GPU and given to the library from pinned host memory, as a program that has read a model
file would.  Every layer has bytes of its own, so a pass streams its weights from HBM.  Hidden rows
are N(0, 1), the state of a residual stream after its RMS norm.
"""
import importlib
import math

import torch

qk = importlib.import_module("qwen-kernel_b200")
syn = qk.synth

TYPES = {"f32": syn.F32, "f16": syn.F16, "q8_0": syn.Q8_0, "q6_k": syn.Q6_K, "iq3_xxs": syn.IQ3_XXS, "iq4_xs": syn.IQ4_XS}
SCALES = {syn.Q8_0: (1e-3, 1e-2), syn.Q6_K: (2e-4, 1e-3), syn.IQ3_XXS: (1e-3, 1e-2), syn.IQ4_XS: (1e-3, 1e-2)}
SCALE_AT = {syn.Q8_0: 0, syn.Q6_K: 208, syn.IQ3_XXS: 0, syn.IQ4_XS: 0}   # byte offset of a block's f16 scale
EPS = 1e-6


def _layers(name, call, tokens, layers, gateup="iq3_xxs", down="iq4_xs", router="f16", experts=256, used=8):
    return {"name": name, "call": call, "tokens": tokens, "layers": layers, "gateup": gateup, "down": down, "router": router,
            "experts": experts, "used": used}


def listed():
    return [
        # one user, one token a step: what a single stream's latency is made of (router in F32, as model files hold it)
        _layers("decode_1", "stack", 1, 24, router="f32"),
        # the server's steady state: 16 slots through the whole 40-layer stack
        _layers("decode_16", "stack", 16, 40),
        # an engine that keeps its activations on the host: rows in, rows out, every step
        _layers("decode_5_host", "stack_host", 5, 24),
        # a full batch of slots, on layers whose down tensors are Q6_K
        _layers("decode_64_q6k", "stack", 64, 12, down="q6_k"),
        # the larger variant (512 experts, top 10, IQ4_XS throughout), called layer by layer between attention blocks
        _layers("step_3_512x10", "step", 3, 8, gateup="iq4_xs", router="f32", experts=512, used=10),
        # a short prompt, or the rest of a long one after its full chunks: layer by layer, just above the decode sizes
        _layers("step_77", "step", 77, 4, router="f32"),
        # a prompt chunk of a common size on the other type mix
        _layers("prefill_600_mix", "prefill", 600, 3, gateup="iq4_xs", down="q6_k"),
        # long prompts in large chunks
        _layers("prefill_4096", "prefill", 4096, 3),
        # a decode step's projections outside the experts, one stream: each weight format in turn
        {"name": "gemv_proj_1", "call": "gemv", "types": "q8_0,q6_k,iq4_xs,iq3_xxs,f16", "M": 4096, "K": 2048, "n": 1, "mats": 4},
        # the same projections for 16 slots
        {"name": "gemv_proj_16", "call": "gemv", "types": "q8_0,q6_k,iq4_xs,iq3_xxs,f16", "M": 4096, "K": 2048, "n": 16, "mats": 2},
        # the head of the model and the greedy pick
        {"name": "head_argmax", "call": "head", "types": "q6_k", "M": 151936, "K": 2048, "n": 1, "mats": 1},
        # a prompt chunk's projections outside the experts
        {"name": "dense_1000", "call": "dense", "types": "q8_0,iq4_xs", "M": 4096, "K": 2048, "n": 1000, "mats": 2},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "gemv", "gemv", "dense"))
    if kind in ("decode", "prefill"):
        wide = rng.random() < 0.25
        c = {"call": rng.choice(("stack", "stack_host", "step") if kind == "decode" else ("prefill", "prefill", "step")),
             "tokens": _log_int(rng, 1, 64) if kind == "decode" else _log_int(rng, 65, 4096),
             "layers": (rng.randint(3, 4) if wide else rng.randint(6, 14)) if kind == "decode" else 2,
             "gateup": rng.choice(("iq3_xxs", "iq3_xxs", "iq4_xs")), "down": rng.choice(("iq4_xs", "iq4_xs", "q6_k")),
             "router": rng.choice(("f32", "f16")), "experts": 512 if wide else 256, "used": 10 if wide else 8}
        return c
    if kind == "gemv":
        t, m, k = rng.choice(("q8_0", "q6_k", "iq4_xs", "iq3_xxs", "f16")), _log_int(rng, 512, 151936), 256 * rng.randint(2, 16)
        n = rng.choice((1, 1, 1, 2, 3, 6, 11, 16))
        return {"call": "gemv", "types": t, "M": m, "K": k, "n": n, "mats": max(1, min(16, int(2e8 / syn.gemv_bytes(TYPES[t], m, k))))}
    return {"call": "dense", "types": rng.choice(("q8_0", "iq4_xs")), "M": 128 * _log_int(rng, 4, 64), "K": 256 * rng.randint(2, 16),
            "n": _log_int(rng, 65, 2048), "mats": 1}


# ------------------------------------------------------------------ what a user's program has in hand

_shared_stream = []


def _stream():
    """The one stream that all states run on (a stream of the caller's, not the default one)."""
    if not _shared_stream:
        _shared_stream.append(torch.cuda.Stream())
    return _shared_stream[0]


def _blocks(gen, ttype, rows, k):
    """rows x k elements of `ttype` as raw ggml bytes on the GPU."""
    nbytes = rows * syn.row_bytes(ttype, k)
    if ttype in (syn.F32, syn.F16):
        w = torch.randn(rows * k, device="cuda", generator=gen) * 0.02
        return (w if ttype == syn.F32 else w.half()).view(torch.uint8)
    b = torch.randint(-(1 << 63), (1 << 63) - 1, (-(-nbytes // 8),), device="cuda", generator=gen, dtype=torch.int64).view(torch.uint8)[:nbytes]
    elems, size = syn.BLOCK[ttype]
    lo, hi = SCALES[ttype]
    d = (torch.rand(nbytes // size, device="cuda", generator=gen) * (hi - lo) + lo).half()
    at = SCALE_AT[ttype]
    b.view(-1, size)[:, at:at + 2] = d.view(torch.uint8).view(-1, 2)
    return b


class State:
    """A library context, its weights and the buffers of one pass."""

    def __init__(self, case, ctx):
        self.case, self.ctx = case, ctx
        ctx.set_stream(_stream().cuda_stream)

    def __del__(self):
        self.ctx.close()


def _layer_state(case, gen):
    dims = syn.Dims(n_expert=case["experts"], n_used=case["used"])
    n, count = case["tokens"], case["layers"]
    s = State(case, qk.Context(dims, n_layer=count, max_tokens=n, device=torch.cuda.current_device()))
    e, f, x = dims.n_embd, dims.n_ff, dims.n_expert
    rt, gt, dt = TYPES[case["router"]], TYPES[case["gateup"]], TYPES[case["down"]]
    shapes = ((rt, x, e), (syn.F32, 1, e), (gt, x * f, e), (gt, x * f, e), (dt, x * e, f), (syn.Q8_0, f, e), (syn.Q8_0, f, e), (syn.Q8_0, e, f))
    staged = [torch.empty(r * syn.row_bytes(t, k), dtype=torch.uint8, pin_memory=True) for t, r, k in shapes]
    for i in range(count):
        for (t, r, k), h in zip(shapes, staged):
            h.copy_(_blocks(gen, t, r, k))
        s.ctx.upload_layer(i, syn.Layer(dims, rt, gt, dt, *[h.numpy() for h in staged]))

    def rows(scale=1.0):
        return torch.randn((count, n, e), device="cuda", generator=gen) * scale

    if case["call"] == "stack_host":
        s.x = torch.empty((count, n, e), pin_memory=True)
        s.x.copy_(rows())
        s.y = torch.empty((count, n, e), pin_memory=True)
    elif case["call"] == "step":
        s.resid, s.attn = rows(), rows(0.3)
        s.w_post, s.w_next = (1 + 0.1 * torch.randn(e, device="cuda", generator=gen) for _ in range(2))
        s.resid_out, s.xn = torch.empty_like(s.resid), torch.empty_like(s.resid)
    else:
        s.x = rows()
        s.y = torch.empty_like(s.x)
    return s


def _matrix_state(case, gen):
    m, k, n = case["M"], case["K"], case["n"]
    s = State(case, qk.Context(syn.Dims(), n_layer=1, max_tokens=1, device=torch.cuda.current_device()))
    s.types = [TYPES[t] for t in case["types"].split(",")] * case["mats"]
    s.x = torch.randn((len(s.types), n, k), device="cuda", generator=gen)
    s.y = torch.empty((len(s.types), n, m), device="cuda")
    s.tok = torch.empty(n, dtype=torch.int32, device="cuda")
    s.w = []
    for i, t in enumerate(s.types):
        w = _blocks(gen, t, m, k)
        if case["call"] == "dense":
            h = torch.empty(w.numel(), dtype=torch.uint8, pin_memory=True)
            h.copy_(w)
            s.ctx.dense_upload(i, t, h.numpy(), m, k)
        else:
            s.w.append(torch.cat([w, w.new_zeros(256)]))   # matrices lie in one buffer with others: the bytes behind one are readable
    return s


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    s = _layer_state(case, gen) if "layers" in case else _matrix_state(case, gen)
    torch.cuda.synchronize()
    return s


def run(s):
    c, ctx = s.case, s.ctx
    call, n = c["call"], c.get("n") or c["tokens"]
    if call == "stack":
        ctx.moe_decode_stack(0, c["layers"], s.x, n, s.y)
        return s.y
    if call == "stack_host":
        ctx.moe_decode_stack_host(0, c["layers"], s.x.data_ptr(), n, s.y.data_ptr())
        return s.y
    if call == "prefill":
        for i in range(c["layers"]):
            ctx.moe_prefill(i, s.x[i], n, s.y[i])
        return s.y
    if call == "step":
        for i in range(c["layers"]):
            ctx.moe_layer_step(i, s.resid[i], s.attn[i], s.w_post, s.w_next, n, s.resid_out[i], s.xn[i], EPS)
        return s.resid_out, s.xn
    if call == "dense":
        for i in range(len(s.types)):
            ctx.dense_gemm(i, s.x[i], n, s.y[i])
        return s.y
    for i, t in enumerate(s.types):
        ctx.gemv(t, s.w[i], s.x[i], s.y[i], c["M"], c["K"], n)
    if call == "head":
        ctx.argmax(s.y[0], n, c["M"], s.tok)
        return s.y, s.tok
    return s.y


def work(case):
    if "layers" in case:
        dims = syn.Dims(n_expert=case["experts"], n_used=case["used"])
        n, e = case["tokens"], dims.n_embd
        distinct = dims.n_expert * (1 - (1 - dims.n_used / dims.n_expert) ** n)   # experts that n independent rows choose, on average
        layer = syn.layer_touched_bytes(dims, TYPES[case["router"]], TYPES[case["gateup"]], TYPES[case["down"]], distinct)
        layer += n * e * 4 * (4 if case["call"] == "step" else 2)
        return {"bytes": case["layers"] * layer, "flops": case["layers"] * n * syn.flops_per_token(dims)}
    m, k, n = case["M"], case["K"], case["n"]
    types = [TYPES[t] for t in case["types"].split(",")] * case["mats"]
    return {"bytes": sum(syn.gemv_bytes(t, m, k, n) for t in types) + (4 * n * (m + 1) if case["call"] == "head" else 0),
            "flops": len(types) * 2 * m * k * n}


def tolerance(case):
    if case["call"] == "dense":
        return {"rel": 6e-3, "max": 4e-2}   # bf16 operands, f32 sums
    if case["call"] == "prefill" or (case["call"] == "step" and case["tokens"] > 64):
        return {"rel": 1.5e-3, "max": 2e-2}   # the tensor-core path: f16 operands, f32 sums
    return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}   # 32-bit throughout
