"""The measured work of this framework: attention calls as a program that serves or trains a model makes them.

`listed()` names one case for each use, `draw(rng)` gives further cases of the same ranges, `prepare` makes what the
program holds before the call (tensors, caches, page tables, output buffers), `run` is one pass through the public
entry points, `work` counts the bytes and operations no implementation can do without.

Inputs are N(0, 1) from the seed, as in this repository's benchmark and tests; lengths that vary inside a batch come
from the case itself (`lengths`), so that a case always means the same sizes.
"""
import importlib
import math
import random

import numpy as np
import torch

THETA = 500000.0
_state = {}


def framework():
    """The package of the tree whose root is the working folder (its folder name is not a Python identifier)."""
    if "fa" not in _state:
        _state["fa"] = importlib.import_module("flat-attention_b200")
    return _state["fa"]


def context():
    """One context for the process, as a program keeps it: device, stream and scratch."""
    if "ctx" not in _state:
        _state["ctx"] = framework().Context(0)
    return _state["ctx"]


# ---- the cases -----------------------------------------------------------------------------------

def listed():
    return [
        # the f32 mode on the grouped shape the reference quotes its own forward numbers on (8 / 2 heads, 512 tokens):
        # small models and numerics work
        dict(name="f32_forward", kind="forward", dtype="f32", layout="projection", B=1, Hq=8, Hkv=2, Nq=512, Nkv=512, D=128,
             causal=True, rope=True, alibi=False),
        # time to first token of one short chat prompt: a fraction of the chip, latency and launches count
        dict(name="prompt_short", kind="forward", dtype="bf16", layout="head_major", B=1, Hq=32, Hkv=8, Nq=333, Nkv=333, D=128,
             causal=True, rope=True, alibi=False),
        # the headline prefill: a batch of four 4096-token prompts
        dict(name="prefill_batch", kind="forward", dtype="bf16", layout="head_major", B=4, Hq=32, Hkv=8, Nq=4096, Nkv=4096, D=128,
             causal=True, rope=True, alibi=False),
        # an encoder: bidirectional multi-head attention in binary16 storage, head_dim 64, a length that is no whole tile
        dict(name="encoder_f16", kind="forward", dtype="f16", layout="head_major", B=8, Hq=16, Hkv=16, Nq=1500, Nkv=1500, D=64,
             causal=False, rope=False, alibi=False),
        # a follow-up turn with the ALiBi bias: new rows against a longer history (rectangular, position offset)
        dict(name="continue_alibi", kind="forward", dtype="bf16", layout="projection", B=2, Hq=32, Hkv=8, Nq=1000, Nkv=3000, D=128,
             causal=True, rope=True, alibi=True),
        # a batch of prompts sorted into length buckets of 256 and padded to the bucket's end
        dict(name="prefill_varlen", kind="varlen", B=16, Hq=32, Hkv=8, N=1024, D=128, lengths=7),
        # one interactive user: a single token against a short paged cache, the smallest call of a serving loop
        dict(name="decode_one", kind="decode_paged", Hq=32, Hkv=8, D=128, page=16, ctx=700),
        # a full serving batch: 64 sequences of 512 to 8192 tokens in a shuffled page pool
        dict(name="decode_batch", kind="decode_batch", S=64, Hq=32, Hkv=8, D=128, page=16, lo=512, hi=8192, lengths=5),
        # few users with long documents in a resident (contiguous) cache
        dict(name="decode_long", kind="decode_resident", dtype="bf16", B=2, Hq=64, Hkv=8, D=128, ctx=60001, capacity=65536),
        # a 32768-token document fed in 2048-token chunks into a growing paged cache
        dict(name="prefill_chunked", kind="chunked", Hq=64, Hkv=8, D=128, N=32768, chunk=2048, page=16, shadow=True),
        # a fine-tuning step on short sequences: forward, then gradients, head_dim 64 and a ragged length
        dict(name="train_short", kind="train", B=2, Hq=16, Hkv=4, N=1000, D=64, causal=True),
        # gradients of a long-context training batch
        dict(name="backward_long", kind="backward", B=2, Hq=32, Hkv=8, N=8192, D=128, causal=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


HEADS = [(8, 2), (16, 4), (16, 16), (32, 8), (64, 8)]
# the most work of one drawn case: attention operations, and bytes of a decode step's cache
MOST_FLOPS = 2.7e12
MOST_CACHE_BYTES = 1.3e9


def draw(rng):
    """One more case of the ranges above."""
    kind = rng.choice(["f32", "prompt", "encoder", "alibi", "varlen", "decode_paged", "decode_batch", "decode_resident",
                       "chunked", "train", "backward"])
    Hq, Hkv = rng.choice(HEADS)
    D = rng.choice([64, 128, 128])
    if kind == "f32":
        Hq, Hkv = rng.choice([(2, 2), (8, 2), (8, 8), (16, 4)])
        n = _log_int(rng, 64, 2048)
        return dict(kind="forward", dtype="f32", layout=rng.choice(["head_major", "projection"]), B=rng.choice([1, 1, 2]), Hq=Hq,
                    Hkv=Hkv, Nq=n, Nkv=n, D=D, causal=rng.random() < 0.7, rope=True, alibi=False)
    if kind == "prompt":
        B, n = rng.choice([1, 1, 2, 4, 8]), _log_int(rng, 64, 8192)
        while 2.0 * B * Hq * n * n * D > MOST_FLOPS:
            n = n * 3 // 4
        return dict(kind="forward", dtype=rng.choice(["bf16", "bf16", "f16"]), layout=rng.choice(["head_major", "projection"]), B=B,
                    Hq=Hq, Hkv=Hkv, Nq=n, Nkv=n, D=D, causal=True, rope=True, alibi=False)
    if kind == "encoder":
        Hq, Hkv = rng.choice([(8, 8), (16, 16), (12, 12)])
        B, n = _log_int(rng, 1, 32), _log_int(rng, 64, 4096)
        while 4.0 * B * Hq * n * n * D > MOST_FLOPS:
            n = n * 3 // 4
        return dict(kind="forward", dtype=rng.choice(["f16", "bf16"]), layout="head_major", B=B, Hq=Hq, Hkv=Hkv, Nq=n, Nkv=n, D=D,
                    causal=False, rope=False, alibi=False)
    if kind == "alibi":
        nkv = _log_int(rng, 256, 8192)
        nq = min(nkv, _log_int(rng, 64, 4096))
        return dict(kind="forward", dtype="bf16", layout="projection", B=rng.choice([1, 2, 4]), Hq=Hq, Hkv=Hkv, Nq=nq, Nkv=nkv, D=D,
                    causal=True, rope=True, alibi=rng.random() < 0.7)
    if kind == "varlen":
        return dict(kind="varlen", B=_log_int(rng, 2, 32), Hq=Hq, Hkv=Hkv, N=_log_int(rng, 256, 4096), D=D,
                    lengths=rng.randrange(1 << 20))
    if kind == "decode_paged":
        return dict(kind="decode_paged", Hq=Hq, Hkv=Hkv, D=D, page=rng.choice([16, 16, 32]), ctx=_log_int(rng, 16, 32768))
    if kind == "decode_batch":
        S, hi = _log_int(rng, 2, 128), _log_int(rng, 128, 16384)
        while 2.0 * S * hi * Hkv * D * 2 > 2 * MOST_CACHE_BYTES:
            S = S * 3 // 4
        return dict(kind="decode_batch", S=S, Hq=Hq, Hkv=Hkv, D=D, page=rng.choice([16, 16, 32, 64]), lo=max(1, hi // 16), hi=hi,
                    lengths=rng.randrange(1 << 20))
    if kind == "decode_resident":
        dtype = rng.choice(["bf16", "bf16", "f32"])
        B, ctx = _log_int(rng, 1, 16), _log_int(rng, 256, 131072)
        while 2.0 * B * ctx * Hkv * D * 4 > MOST_CACHE_BYTES:
            ctx = ctx * 3 // 4
        return dict(kind="decode_resident", dtype=dtype, B=B, Hq=Hq, Hkv=Hkv, D=D, ctx=ctx, capacity=ctx + rng.randrange(0, 512))
    if kind == "chunked":
        n = _log_int(rng, 1024, 16384)
        chunk = rng.choice([1024, 2048, 4096])
        return dict(kind="chunked", Hq=Hq, Hkv=Hkv, D=D, N=n, chunk=chunk, page=rng.choice([16, 32]), shadow=rng.random() < 0.5)
    B, n = rng.choice([1, 2, 4]), _log_int(rng, 128, 2048 if kind == "train" else 8192)
    while 5.0 * B * Hq * n * n * D > MOST_FLOPS:
        n = n * 3 // 4
    return dict(kind=kind, B=B, Hq=Hq, Hkv=Hkv, N=n, D=D, causal=rng.random() < 0.8)


# ---- states and passes ---------------------------------------------------------------------------

def _lengths(case):
    """Lengths of the batch's sequences, drawn from the case's own seed."""
    rng = random.Random(case["lengths"])
    if case["kind"] == "varlen":
        bucket = (case["N"] - 1) // 256 * 256
        return [rng.randint(bucket + 1, case["N"]) for _ in range(case["B"])]
    return [rng.randint(case["lo"], case["hi"]) for _ in range(case["S"])]


def _randn(g, dtype, *size):
    return torch.randn(*size, generator=g, device="cuda", dtype=torch.float32).to(dtype)


class _DeviceArray:
    """A buffer of a cache as an array other libraries can view; the view keeps the cache alive."""

    def __init__(self, cache, ptr, count, typestr):
        self.cache = cache
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3, "strides": None}


def _view(cache, buffer, dtype):
    size = 4 if dtype == torch.float32 else 2
    raw = torch.as_tensor(_DeviceArray(cache, buffer.ptr, buffer.bytes // size, "<i%d" % size), device="cuda")
    return raw.view(dtype)


def prepare(case, seed):
    fa, ctx = framework(), context()
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    D, Hq, Hkv = case["D"], case["Hq"], case["Hkv"]
    s = dict(case)
    s["ctx_obj"] = ctx
    if kind == "forward":
        code, dtype = {"f32": (fa.F32, torch.float32), "bf16": (fa.BF16, torch.bfloat16), "f16": (fa.F16, torch.float16)}[case["dtype"]]
        B, Nq, Nkv = case["B"], case["Nq"], case["Nkv"]
        layout = fa.HEAD_MAJOR if case["layout"] == "head_major" else fa.PROJECTION
        s["q"], s["k"], s["v"] = (_randn(g, dtype, B * n * h * D) for n, h in ((Nq, Hq), (Nkv, Hkv), (Nkv, Hkv)))
        s["shape"] = fa.shape(B, Hq, Hkv, Nq, Nkv, D, Nkv - Nq)
        s["config"] = fa.config(case["causal"])
        s["rotary"] = fa.rotary(THETA, Nkv - Nq, 0)
        s["code"] = code
        s["slopes"] = [2.0 ** (-8.0 * (h + 1) / Hq) for h in range(Hq)]
        s["out"] = ctx.create_output_buffer(code, s["shape"])
        s["views"] = ctx.split_output(s["out"], code, s["shape"], layout)
    elif kind == "varlen":
        B, N = case["B"], case["N"]
        s["q"], s["k"], s["v"] = (_randn(g, torch.bfloat16, B * N * h * D) for h in (Hq, Hkv, Hkv))
        s["shape"] = fa.shape(B, Hq, Hkv, N, N, D)
        s["config"], s["rotary"] = fa.config(True), fa.rotary(THETA, 0)
        s["sequences"] = [fa.VarlenSequence(n, n, 0, 0) for n in _lengths(case)]
        s["out"] = ctx.create_output_buffer(fa.BF16, s["shape"])
        s["views"] = ctx.split_output(s["out"], fa.BF16, s["shape"], fa.PROJECTION)
    elif kind == "decode_paged":
        n, page = case["ctx"], case["page"]
        cache = fa.CudaPagedKvCache(ctx, fa.BF16, page, (n + page - 1) // page + 1, Hkv, D)
        k, v = (_randn(g, torch.bfloat16, n * Hkv * D) for _ in range(2))
        cache.record_append(k, v, n)
        s["cache"], s["table"], s["k"], s["v"] = cache, cache.table(), cache.k_buffer(), cache.v_buffer()
        s["q"] = _randn(g, torch.bfloat16, Hq * D)
        s["config"] = fa.config(True)
        s["out"] = ctx.create_decode_output_buffer(fa.BF16, 1, Hq, D)
        s["views"] = ctx.split_decode_output(s["out"], fa.BF16, 1, Hq, D)
    elif kind == "decode_batch":
        S, page = case["S"], case["page"]
        lens = np.array(_lengths(case), np.int32)
        pages = (lens + page - 1) // page
        pool, widest = int(pages.sum()), int(pages.max())
        shuffled = np.random.default_rng(seed).permutation(pool).astype(np.int32)
        tables = np.zeros((S, widest), np.int32)
        at = 0
        for i, n in enumerate(pages):
            tables[i, :n] = shuffled[at:at + n]
            at += n
        s["host"] = (tables, lens, (lens - 1).astype(np.int32))
        s["device"] = tuple(torch.from_numpy(x).cuda() for x in s["host"])
        s["pool"], s["widest"] = pool, widest
        s["k"], s["v"] = (_randn(g, torch.bfloat16, pool * page * Hkv * D) for _ in range(2))
        s["q"] = _randn(g, torch.bfloat16, S * Hq * D)
        s["config"] = fa.config(True)
        s["out"] = ctx.create_decode_output_buffer(fa.BF16, S, Hq, D)
        s["views"] = ctx.split_decode_output(s["out"], fa.BF16, S, Hq, D)
    elif kind == "decode_resident":
        code, dtype = (fa.F32, torch.float32) if case["dtype"] == "f32" else (fa.BF16, torch.bfloat16)
        B, n = case["B"], case["ctx"]
        cache = fa.CudaResidentKvCache(ctx, code, B, Hkv, case["capacity"], D)
        k, v = (_randn(g, dtype, B * n * Hkv * D) for _ in range(2))
        cache.record_append(k, v, n)
        s["cache"], s["k"], s["v"] = cache, cache.k_buffer(), cache.v_buffer()
        s["q"] = _randn(g, dtype, B * Hq * D)
        s["config"], s["code"] = fa.config(True), code
        s["out"] = ctx.create_decode_output_buffer(code, B, Hq, D)
        s["views"] = ctx.split_decode_output(s["out"], code, B, Hq, D)
    elif kind == "chunked":
        N, chunk, page = case["N"], case["chunk"], case["page"]
        cache = fa.CudaPagedKvCache(ctx, fa.BF16, page, (N + page - 1) // page, Hkv, D)
        if case["shadow"]:
            cache.enable_prefill_shadow()
        q = _randn(g, torch.bfloat16, N, Hq * D)
        k, v = (_randn(g, torch.bfloat16, N, Hkv * D) for _ in range(2))
        s["cache"], s["config"] = cache, fa.config(True)
        s["chunks"], s["views"] = [], []
        for start in range(0, N, chunk):
            n = min(chunk, N - start)
            shape = fa.shape(1, Hq, Hkv, n, n, D)
            out = ctx.create_output_buffer(fa.BF16, shape)
            s["chunks"].append((n, q[start:start + n], k[start:start + n], v[start:start + n], out))
            s["views"].append(ctx.split_output(out, fa.BF16, shape, fa.PROJECTION))
        s["views"].append(tuple(_view(cache, b, torch.bfloat16) for b in (cache.k_buffer(), cache.v_buffer())))
    else:  # train, backward: the packed buffers of the backward call; the forward writes its [O | LSE] straight into them
        B, N = case["B"], case["N"]
        s["shape"], s["config"] = fa.shape(B, Hq, Hkv, N, N, D), fa.config(case["causal"])
        L = fa.backward_layout(fa.BF16, s["shape"])
        packed = ctx.empty_bytes(L.input_bytes)
        for at, count in ((L.q_offset, L.q_elements), (L.k_offset, L.kv_elements), (L.v_offset, L.kv_elements),
                          (L.d_out_offset, L.q_elements)):
            packed[at:at + 2 * count].view(torch.bfloat16).copy_(_randn(g, torch.bfloat16, count))
        s["q"], s["k"], s["v"] = (packed[at:at + 2 * n].view(torch.bfloat16) for at, n in
                                  ((L.q_offset, L.q_elements), (L.k_offset, L.kv_elements), (L.v_offset, L.kv_elements)))
        s["fwd"] = packed[L.out_offset:]
        s["packed"], s["grads"] = packed, ctx.empty_bytes(L.output_bytes)
        grads = tuple(s["grads"][at:at + 4 * n].view(torch.float32) for at, n in
                      ((L.dq_offset, L.q_elements), (L.dk_offset, L.kv_elements), (L.dv_offset, L.kv_elements)))
        s["views"] = grads
        if kind == "train":
            s["views"] = (ctx.split_output(s["fwd"], fa.BF16, s["shape"]), grads)
        else:
            ctx.forward_grouped(fa.BF16, s["shape"], s["config"], s["q"], s["k"], s["v"], s["fwd"])
    return s


def run(s):
    fa, ctx, kind = framework(), s["ctx_obj"], s["kind"]
    if kind == "forward":
        args = (s["q"], s["k"], s["v"], s["out"])
        if s["alibi"]:
            ctx.forward_projection_rope_asymmetric_alibi(s["code"], s["shape"], s["config"], s["rotary"], s["slopes"],
                                                         s["Nkv"] - s["Nq"], 0, *args)
        elif s["layout"] == "projection":
            ctx.forward_projection_rope_asymmetric(s["code"], s["shape"], s["config"], s["rotary"], *args)
        elif s["rope"]:
            ctx.forward_grouped_rope(s["code"], s["shape"], s["config"], s["rotary"], *args)
        else:
            ctx.forward_grouped(s["code"], s["shape"], s["config"], *args)
    elif kind == "varlen":
        ctx.forward_projection_rope_varlen(fa.BF16, s["shape"], s["config"], s["rotary"], s["sequences"], s["q"], s["k"], s["v"],
                                           s["out"])
    elif kind == "decode_paged":
        ctx.decode_paged(fa.BF16, s["table"], s["Hq"], s["Hkv"], s["D"], s["config"], THETA, s["ctx"] - 1, s["q"], s["k"], s["v"],
                         s["out"])
    elif kind == "decode_batch":
        ctx.decode_paged_batched(fa.BF16, s["S"], s["Hq"], s["Hkv"], s["D"], s["page"], s["pool"], s["widest"], *s["device"],
                                 *s["host"], s["config"], THETA, s["q"], s["k"], s["v"], s["out"])
    elif kind == "decode_resident":
        ctx.decode_resident(s["code"], s["B"], s["Hq"], s["Hkv"], s["D"], s["ctx"], s["capacity"], s["config"], THETA, s["ctx"] - 1,
                            s["q"], s["k"], s["v"], s["out"])
    elif kind == "chunked":
        s["cache"].reset()
        for n, q, k, v, out in s["chunks"]:
            ctx.chunked_prefill_paged(s["cache"], s["Hq"], n, s["config"], THETA, 0, q, k, v, out)
    else:
        if kind == "train":
            ctx.forward_grouped(fa.BF16, s["shape"], s["config"], s["q"], s["k"], s["v"], s["fwd"])
        ctx.backward_grouped(fa.BF16, s["shape"], s["config"], s["packed"], s["grads"])
    return s["views"]


# ---- what a pass cannot do without ---------------------------------------------------------------

def _pairs(nq, nkv, causal):
    """Visible (query, key) pairs of one head; the queries are the last nq positions of nkv."""
    return nq * nkv - (nq * (nq - 1) // 2 if causal else 0)


def work(case):
    kind = case["kind"]
    D, Hq, Hkv = case["D"], case["Hq"], case["Hkv"]
    if kind == "forward":
        es = 4 if case["dtype"] == "f32" else 2
        B, nq, nkv = case["B"], case["Nq"], case["Nkv"]
        return {"bytes": B * D * es * (2 * nq * Hq + 2 * nkv * Hkv) + 4 * B * Hq * nq,
                "flops": 4 * B * Hq * D * _pairs(nq, nkv, case["causal"])}
    if kind == "varlen":  # live rows in; the whole padded output is written
        lens = _lengths(case)
        return {"bytes": 2 * D * sum(lens) * (Hq + 2 * Hkv) + case["B"] * case["N"] * Hq * (2 * D + 4),
                "flops": 4 * Hq * D * sum(_pairs(n, n, True) for n in lens)}
    if kind in ("decode_paged", "decode_resident", "decode_batch"):
        es = 4 if case.get("dtype") == "f32" else 2
        rows = case.get("S", case.get("B", 1))
        tokens = sum(_lengths(case)) if kind == "decode_batch" else rows * case["ctx"]
        return {"bytes": 2 * tokens * Hkv * D * es + rows * Hq * (2 * D * es + 4), "flops": 4 * tokens * Hq * D}
    if kind == "chunked":  # Q, K, V in; O, LSE and the cache out
        N = case["N"]
        return {"bytes": 2 * N * D * (2 * Hq + 4 * Hkv) + 4 * N * Hq, "flops": 4 * Hq * D * _pairs(N, N, True)}
    B, N = case["B"], case["N"]
    pairs = B * Hq * D * _pairs(N, N, case["causal"])
    grads = 4 * B * N * D * (Hq + 2 * Hkv)
    if kind == "backward":  # Q, K, V, dO, O, LSE in; f32 gradients out
        return {"bytes": 2 * B * N * D * (3 * Hq + 2 * Hkv) + 4 * B * N * Hq + grads, "flops": 10 * pairs}
    return {"bytes": 2 * B * N * D * (3 * Hq + 2 * Hkv) + 4 * B * N * Hq + grads, "flops": 14 * pairs}


def tolerance(case):
    """About four times the distance of the present outputs from the same pass in 64 bits (2-norm, and the largest element)."""
    dtype = case.get("dtype", "bf16")
    if dtype == "f32":
        return {"rel": 1e-5, "max": 1e-4}
    if dtype == "f16":
        return {"rel": 2e-3, "max": 3e-2}
    if case["kind"] in ("train", "backward"):  # measured 1.9e-3 and 1e-1: early rows have few terms and small gradients
        return {"rel": 1e-2, "max": 4e-1}
    return {"rel": 1.2e-2, "max": 1.6e-1}  # measured up to 2.9e-3 and 4e-2
