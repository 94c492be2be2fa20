"""The work that a user of this library has it do, as timed cases through its public entry points.

Families (the key "work" of a case):

  step      one decode step of a batch: q rotated, the new token of every sequence written into its cache, the batch attended
            over the caches (`ops.rope_apply` + `ops.decode_append`)
  hoststep  the same for a host that keeps the step's q / k / v and its result in pinned memory (`ops.DecodeStep`)
  prompt    a batch of prompts: q and k rotated, K / V quantised into the caches, causal attention
  chunk     one chunk of a long prompt behind a cached prefix, through the cache object: `LayerKVCache.update`, `.get`, attention
  qprompt   a prompt through a block of 3 gated-DeltaNet layers and 1 gated full-attention layer (`ops.qwen_block_forward`)
  qstep     one decode step of a batch through the same block
  tensor    a whole tensor quantised blockwise and dequantised again (weights or cache images that are kept quantised)

The caches of all families but "chunk" are the caller's own device buffers behind a `KVView`, so a case can return them.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from hyprstream_b200 import ffi, kv_cache as kc, ops

KINDS = {"bf16": ffi.KV_BF16, "int8": ffi.KV_INT8, "nf4": ffi.KV_NF4, "fp4": ffi.KV_FP4}
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
PAGE = 256                               # tokens of a pool page
GDN_LAYERS, NK, NV, HD, TAPS = 3, 16, 32, 128, 4  # the block: DeltaNet heads, head dim, conv taps
QHQ, QHKV, QD, QROT = 16, 2, 256, 64     # ... and its full-attention layer


# ------------------------------------------------------------------------------------------------ the cases
def listed() -> list:
    llama = {"hq": 32, "hkv": 8, "d": 128}
    return [
        # the smallest call: one chat, an unquantised cache of 4096 tokens (the default storage)
        {"name": "step_bf16_1x4096", "work": "step", "kind": "bf16", "block": 64, "f16": False, "n": 1, "lo": 4096, "hi": 4096, "lens_seed": 1,
         "paged": False, "rope": True, **llama},
        # a serving batch, ragged contexts, int8 cache with one f16 scale per head row; keys arrive rotated
        {"name": "step_int8_32_ragged", "work": "step", "kind": "int8", "block": 128, "f16": True, "n": 32, "lo": 512, "hi": 8192, "lens_seed": 1,
         "paged": False, "rope": False, **llama},
        # a small batch of an engine whose tensors are in host memory, int8 cache in the default layout, pages of a shared pool
        {"name": "hoststep_int8_paged_7", "work": "hoststep", "kind": "int8", "block": 64, "f16": False, "n": 7, "lo": 17, "hi": 3000, "lens_seed": 2,
         "paged": True, "rope": True, **llama},
        # long contexts in a 4-bit cache
        {"name": "step_nf4_4x131072", "work": "step", "kind": "nf4", "block": 64, "f16": True, "n": 4, "lo": 131072, "hi": 131072, "lens_seed": 3,
         "paged": False, "rope": True, **llama},
        # a serving batch over the unquantised paged pool
        {"name": "step_bf16_paged_16", "work": "step", "kind": "bf16", "block": 64, "f16": False, "n": 16, "lo": 100, "hi": 6000, "lens_seed": 4,
         "paged": True, "rope": True, **llama},
        # the largest prompt batch, written into an int8 cache
        {"name": "prompt_int8_8x8192", "work": "prompt", "kind": "int8", "block": 128, "f16": True, "n": 8, "t": 8192, "paged": False, **llama},
        # two mid-size prompts of an odd length at head_dim 64, 4-bit cache
        {"name": "prompt_nf4_d64_2x1531", "work": "prompt", "kind": "nf4", "block": 64, "f16": False, "n": 2, "t": 1531, "paged": False, "hq": 32,
         "hkv": 8, "d": 64},
        # a chunk of a long prompt behind a cached prefix, the cache object's own calls
        {"name": "chunk_int8_1000_at_3333", "work": "chunk", "kind": "int8", "block": 64, "f16": False, "t": 1000, "prefix": 3333, "paged": False, **llama},
        # the hybrid block: long prompts, a large decode batch at long contexts, a small decode batch
        {"name": "qprompt_4x32768", "work": "qprompt", "n": 4, "t": 32768, "block": 128, "f16": True, "carried": False},
        {"name": "qstep_64x32768", "work": "qstep", "n": 64, "lo": 32768, "hi": 32768, "lens_seed": 5, "block": 128, "f16": True},
        {"name": "qstep_3_ragged", "work": "qstep", "n": 3, "lo": 300, "hi": 3000, "lens_seed": 6, "block": 128, "f16": True},
        # a tensor kept in 4 bits: an odd number of elements, the last block cut short
        {"name": "tensor_nf4_bf16_20M", "work": "tensor", "kind": "nf4", "block": 64, "f16": False, "dtype": "bf16", "elems": 20_000_003},
    ]


def _log(rng, lo: int, hi: int) -> int:
    """An integer of [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _storage(rng) -> dict:
    kind = rng.choice(["bf16", "bf16", "int8", "int8", "int8", "nf4", "nf4", "fp4"])
    block, f16 = rng.choice([(64, False), (128, True), (64, True)]) if kind == "int8" else (64, kind != "bf16" and rng.random() < 0.5)
    return {"kind": kind, "block": block, "f16": f16}


def _heads(rng, storage: dict) -> dict:
    """Mostly 32 / 8 x 128; also 16 / 2 x 256, one kv head per query head, and head_dim 64."""
    hq, hkv, d = rng.choice([(32, 8, 128)] * 5 + [(16, 2, 256)] * 2 + [(8, 8, 128), (32, 8, 64)])
    if d == 64 and storage["block"] > 64:
        hq, hkv, d = 32, 8, 128
    return {"hq": hq, "hkv": hkv, "d": d}


def draw(rng) -> dict:
    work = rng.choice(["step", "step", "step", "hoststep", "prompt", "prompt", "chunk", "qprompt", "qstep", "tensor"])
    if work in ("step", "hoststep"):
        s = _storage(rng)
        n = _log(rng, 1, 64 if work == "step" else 32)
        longest = 131072 if s["kind"] in ("nf4", "fp4") else 65536
        hi = _log(rng, 40, min(longest, 524288 // n) if work == "step" else 8192)
        lo = hi if rng.random() < 0.2 else max(1, int(hi * rng.uniform(0.02, 0.9)))
        return {"work": work, **s, "n": n, "lo": lo, "hi": hi, "lens_seed": rng.randrange(1 << 20), "paged": rng.random() < 0.4,
                "rope": rng.random() < 0.7, **_heads(rng, s)}
    if work == "prompt":
        s = _storage(rng)
        t = _log(rng, 16, 8192)
        return {"work": work, **s, "n": _log(rng, 1, max(1, min(8, 65536 // t))), "t": t, "paged": rng.random() < 0.4, **_heads(rng, s)}
    if work == "chunk":
        s = _storage(rng)
        return {"work": work, **s, "t": _log(rng, 2, 2048), "prefix": _log(rng, 30, 16384), "paged": rng.random() < 0.4, **_heads(rng, s)}
    if work == "qprompt":
        t = _log(rng, 20, 32768)
        return {"work": work, "n": _log(rng, 1, max(1, min(4, 131072 // t))), "t": t, "block": rng.choice([64, 128]), "f16": rng.random() < 0.6,
                "carried": rng.random() < 0.3}
    if work == "qstep":
        n = _log(rng, 1, 64)
        hi = _log(rng, 40, 32768)
        return {"work": work, "n": n, "lo": max(1, int(hi * rng.uniform(0.05, 1.0))), "hi": hi, "lens_seed": rng.randrange(1 << 20),
                "block": rng.choice([64, 128]), "f16": rng.random() < 0.6}
    kind = rng.choice(["int8", "nf4", "fp4"])
    return {"work": "tensor", "kind": kind, "block": rng.choice([64, 64, 128, 256]), "f16": rng.random() < 0.3,
            "dtype": rng.choice(["bf16", "bf16", "f16", "f32"]), "elems": _log(rng, 5000, 67_108_864)}


def _lens(case: dict) -> list:
    """Attended lengths of a step, the new token included: the case's own, whatever the seed of the inputs."""
    if case["lo"] == case["hi"]:
        return [case["lo"]] * case["n"]
    return [int(x) for x in np.random.default_rng(case["lens_seed"]).integers(case["lo"], case["hi"] + 1, size=case["n"])]


# ------------------------------------------------------------------------------------------------ inputs
class _Gen:
    """N(0, 1) values from a seed, on the GPU."""

    def __init__(self, seed: int):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.g = torch.Generator(device=self.dev).manual_seed(int(seed) % (1 << 62))

    def __call__(self, *shape) -> torch.Tensor:
        return torch.randn(*shape, device=self.dev, generator=self.g)

    def b(self, *shape) -> torch.Tensor:
        return self(*shape).bfloat16()

    def rand(self, *shape) -> torch.Tensor:
        return torch.rand(*shape, device=self.dev, generator=self.g)


class _Cache:
    """Device buffers of one layer's cache for a batch and the `KVView` over them: one run of tokens per sequence, or pages of a
    shared pool in shuffled order."""

    def __init__(self, rnd: _Gen, kind: int, block: int, f16: bool, hkv: int, d: int, lens: list, paged: bool):
        dev = rnd.dev
        if paged:
            page = PAGE
            need = [(l + PAGE - 1) // PAGE for l in lens]
            pages, pps = sum(need), max(need)
            order = torch.randperm(pages, device=dev, generator=rnd.g)
        else:
            page = (max(lens) + 1023) // 1024 * 1024  # caches grow by 1024 tokens
            need, pages, pps = [1] * len(lens), len(lens), 1
            order = torch.arange(pages, device=dev)
        row = {ffi.KV_BF16: 2 * d, ffi.KV_INT8: d}.get(kind, d // 2)
        self.k, self.v = (torch.zeros(pages, page, hkv, row, dtype=torch.uint8, device=dev) for _ in range(2))
        self.tensors = [self.k, self.v]
        if kind != ffi.KV_BF16:
            sdt = torch.float16 if f16 else torch.float32
            self.tensors += [torch.zeros(pages, page, hkv, d // block, dtype=sdt, device=dev) for _ in range(2)]
        slot = torch.zeros(len(lens), pps, dtype=torch.int64, device=dev)  # page number of (sequence, page of the sequence)
        at = 0
        for s, m in enumerate(need):
            slot[s, :m] = order[at:at + m]
            at += m
        self.tables = [(t.data_ptr() + slot * (t.stride(0) * t.element_size())).contiguous() for t in self.tensors]
        tp = [t.data_ptr() for t in self.tables] + [None] * (4 - len(self.tables))
        self.stride = pps * 8
        self.view = ffi.KVView(kind, ffi.SCALE_F16 if f16 else ffi.SCALE_F32, block, hkv, d, page, pps, 0, *tp)
        self.bf16 = kind == ffi.KV_BF16

    def fill(self, rnd: _Gen, lens: list) -> None:
        """N(0, 1) keys and values for the first lens[s] tokens of every sequence, written by the library."""
        hkv, d = self.view.n_kv_heads, self.view.head_dim
        for s, l in enumerate(lens):
            sub = ffi.KVView.from_buffer_copy(self.view)
            for f in ("k_pages", "v_pages", "k_scale_pages", "v_scale_pages"):
                if getattr(self.view, f):
                    setattr(sub, f, getattr(self.view, f) + s * self.stride)
            for t0 in range(0, l, 65536):
                m = min(65536, l - t0)
                ops.kv_quantize_write(sub, rnd.b(1, m, hkv, d), rnd.b(1, m, hkv, d), torch.full((1,), t0, dtype=torch.int32, device=rnd.dev))

    def out(self) -> list:
        return [t.view(torch.bfloat16) for t in self.tensors] if self.bf16 else list(self.tensors)


def _i32(values, dev) -> torch.Tensor:
    return torch.tensor(values, dtype=torch.int32, device=dev)


def _rope_tables(rotary: int, n: int, dev, base: float = 500000.0):
    inv = base ** (-torch.arange(0, rotary, 2, device=dev, dtype=torch.float64) / rotary)
    ang = torch.arange(n, device=dev, dtype=torch.float64)[:, None] * inv[None, :]
    return torch.sin(ang).bfloat16(), torch.cos(ang).bfloat16()


def _gdn_layers(rnd: _Gen) -> list:
    conv = (2 * NK + NV) * HD
    return [ops.GdnLayer((rnd(conv, 1, TAPS) * 0.5).bfloat16(), torch.log(rnd.rand(NV) + 1e-3), rnd(NV) * 0.3, 1.0 + 0.1 * rnd(HD), NK, NV)
            for _ in range(GDN_LAYERS)]


def _block(rnd: _Gen, case: dict, b: int, t: int, lens: list, carried: bool, fill: list) -> dict:
    """Weights, projection outputs, states and cache of the hybrid block for b sequences of t new tokens."""
    dev, conv = rnd.dev, (2 * NK + NV) * HD
    start = [l - t for l in lens]
    sin, cos = _rope_tables(QROT, max(lens) + 1, dev)
    layers, attn = _gdn_layers(rnd), ops.QwenAttnLayer(0.1 * rnd(QD), 0.1 * rnd(QD), sin, cos, QROT, QHQ, QHKV, QD)
    cache = _Cache(rnd, ffi.KV_INT8, case["block"], case["f16"], QHKV, QD, lens, False)
    cache.fill(rnd, fill)
    gin = []
    for l in layers:
        x, z, a, bb = rnd.b(b, t, conv), rnd.b(b, t, NV, HD), rnd.b(b, t, NV), rnd.b(b, t, NV)
        cs, rs = l.new_states(b, dev)
        if carried:
            cs, rs = rnd.b(b, conv, TAPS - 1), 0.1 * rnd(b, NV, HD, HD)
        gin.append((x, z, a, bb, cs, rs))
    dst = _i32(start, dev)
    pos = (dst[:, None] + torch.arange(t, device=dev, dtype=torch.int32)[None, :]).reshape(-1).contiguous()
    ain = (rnd.b(b * t, QHQ * 2 * QD), rnd.b(b * t, QHKV * QD), rnd.b(b, t, QHKV, QD), cache.view, pos, dst, _i32(lens, dev))
    ws = torch.empty(max(layers[0].workspace_bytes(b, t), attn.workspace_bytes(b, t)), dtype=torch.uint8, device=dev)
    return {"layers": layers, "gin": gin, "attn": attn, "ain": ain, "cache": cache, "b": b, "t": t, "has": carried, "ws": ws, "dev": dev}


def prepare(case: dict, seed: int) -> dict:
    rnd, w = _Gen(seed), case["work"]
    dev = rnd.dev
    if w == "tensor":
        # channels of very different size, as activations have them
        n = case["elems"]
        x = rnd(n) * torch.exp(rnd((n + 127) // 128)).repeat_interleave(128)[:n]
        return {"work": w, "x": x.to(DTYPES[case["dtype"]]), "kind": KINDS[case["kind"]], "block": case["block"],
                "sd": ffi.SCALE_F16 if case["f16"] else ffi.SCALE_F32}
    if w == "qstep":
        lens = _lens(case)
        return {"work": w, **_block(rnd, case, case["n"], 1, lens, True, [l - 1 for l in lens])}
    if w == "qprompt":
        return {"work": w, **_block(rnd, case, case["n"], case["t"], [case["t"]] * case["n"], case["carried"], [])}
    hq, hkv, d, kind = case["hq"], case["hkv"], case["d"], KINDS[case["kind"]]
    rotary = 64 if d == 256 else d
    if w == "chunk":
        t, p = case["t"], case["prefix"]
        sd = ffi.SCALE_F16 if case["f16"] else ffi.SCALE_F32
        if case["paged"]:
            pool = kc.BlockPool((p + t + PAGE - 1) // PAGE + 2, hkv, d, dev, kind=kind, block=case["block"], scale_dtype=sd)
            cache = kc.LayerKVCache.new_paged(32768, pool, owner=1)
        else:
            cache = kc.LayerKVCache(32768, kc.KVQuantType(kind), hkv, d, dev, block=case["block"], scale_dtype=sd)
        cache._ensure_capacity(p + t)
        cache.update(rnd.b(1, p, hkv, d), rnd.b(1, p, hkv, d), 0)
        return {"work": w, "cache": cache, "q": rnd.b(1, t, hq, d), "k": rnd.b(1, t, hkv, d), "v": rnd.b(1, t, hkv, d), "prefix": p}
    n = case["n"]
    if w == "prompt":
        t = case["t"]
        cache = _Cache(rnd, kind, case["block"], case["f16"], hkv, d, [t] * n, case["paged"])
        sin, cos = _rope_tables(rotary, t, dev)
        return {"work": w, "cache": cache, "q": rnd.b(n * t, hq, d), "k": rnd.b(n * t, hkv, d), "v": rnd.b(n, t, hkv, d), "sin": sin, "cos": cos,
                "rotary": rotary, "pos": torch.arange(t, dtype=torch.int32, device=dev).repeat(n), "dst": torch.zeros(n, dtype=torch.int32, device=dev),
                "n": n, "t": t}
    lens = _lens(case)
    cache = _Cache(rnd, kind, case["block"], case["f16"], hkv, d, lens, case["paged"])
    cache.fill(rnd, [l - 1 for l in lens])
    st = {"work": w, "cache": cache, "lens": _i32(lens, dev), "rotary": 0, "sin": None, "cos": None}
    if case["rope"]:
        st["sin"], st["cos"] = _rope_tables(rotary, max(lens) + 1, dev)
        st["rotary"] = rotary
    if w == "hoststep":
        st["step"] = ops.DecodeStep(cache.view, n, hq, dev)
        for h, shape in (("q_host", (n, hq, d)), ("k_host", (n, hkv, d)), ("v_host", (n, hkv, d))):
            getattr(st["step"], h).copy_(rnd.b(*shape))
        return st
    st["q"], st["k"], st["v"] = rnd.b(n, hq, d), rnd.b(n, 1, hkv, d), rnd.b(n, 1, hkv, d)
    st["pos"] = st["lens"] - 1
    return st


# ------------------------------------------------------------------------------------------------ one pass
def run(st: dict):
    w = st["work"]
    if w == "step":
        q = st["q"] if st["sin"] is None else ops.rope_apply(st["q"], st["sin"], st["cos"], st["pos"], st["rotary"])
        out = ops.decode_append(q, st["k"], st["v"], st["cache"].view, None, st["lens"], sin=st["sin"], cos=st["cos"], rotary_dim=st["rotary"])
        return [out] + st["cache"].out()
    if w == "hoststep":
        out = st["step"].run(None, st["lens"], st["sin"], st["cos"], st["rotary"])
        return [out] + st["cache"].out()
    if w == "prompt":
        n, t = st["n"], st["t"]
        q = ops.rope_apply(st["q"], st["sin"], st["cos"], st["pos"], st["rotary"])
        k = ops.rope_apply(st["k"], st["sin"], st["cos"], st["pos"], st["rotary"])
        k = k.view(n, t, *k.shape[1:])
        ops.kv_quantize_write(st["cache"].view, k, st["v"], st["dst"])
        out = ops.prefill_attention(q.view(n, t, *q.shape[1:]), k, st["v"])
        return [out] + st["cache"].out()
    if w == "chunk":
        st["cache"].update(st["k"], st["v"], st["prefix"])
        k, v = st["cache"].get()
        return [ops.prefill_attention(st["q"], k, v), k, v]
    if w in ("qprompt", "qstep"):
        ys, out = ops.qwen_block_forward(st["layers"], st["gin"], st["attn"], st["ain"], st["has"], st["b"], st["t"], st["dev"], workspace=st["ws"])
        return ys + [out] + [s for g in st["gin"] for s in g[4:6]] + st["cache"].out()
    codes, absmax = ops.quantize_blockwise(st["x"], st["kind"], st["block"], st["sd"])
    return [codes, absmax, ops.dequantize_blockwise(codes, absmax, st["kind"], st["x"].numel(), st["block"], st["x"].dtype)]


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _token_bytes(kind: str, block: int, f16: bool, hkv: int, d: int) -> int:
    """K + V of one cached token as stored."""
    if kind == "bf16":
        return 4 * hkv * d
    return 2 * hkv * ((d if kind == "int8" else d // 2) + d // block * (2 if f16 else 4))


def _causal_pairs(t: int, prefix: int = 0) -> int:
    return t * prefix + t * (t + 1) // 2


def work(case: dict) -> dict:
    w = case["work"]
    if w == "tensor":
        n, esz = case["elems"], 4 if case["dtype"] == "f32" else 2
        stored = (n if case["kind"] == "int8" else (n + 1) // 2) + (n + case["block"] - 1) // case["block"] * (2 if case["f16"] else 4)
        return {"bytes": 2 * n * esz + 2 * stored, "flops": 0}
    if w in ("qstep", "qprompt"):
        b, t = case["n"], case.get("t", 1)
        lens = _lens(case) if w == "qstep" else [t] * b
        tok = _token_bytes("int8", case["block"], case["f16"], QHKV, QD)
        conv = (2 * NK + NV) * HD
        states = b * (NV * HD * HD * 4 + conv * (TAPS - 1) * 2) * (1 if w == "qprompt" and not case["carried"] else 2)
        gdn = states + b * t * (conv * 2 + 2 * NV * 2 + 2 * NV * HD * 2)
        attn = b * t * (QHQ * 2 * QD * 2 + 2 * QHKV * QD * 2 + QHQ * QD * 2 + tok)
        pairs = b * _causal_pairs(t) if w == "qprompt" else sum(lens)
        attn += sum(lens) * tok if w == "qstep" else 0
        return {"bytes": GDN_LAYERS * gdn + attn, "flops": 4 * pairs * QHQ * QD + GDN_LAYERS * b * t * NV * 6 * HD * HD}
    hq, hkv, d = case["hq"], case["hkv"], case["d"]
    tok = _token_bytes(case["kind"], case["block"], case["f16"], hkv, d)
    if w in ("step", "hoststep"):
        lens = _lens(case)
        return {"bytes": sum(lens) * tok + case["n"] * (4 * hq * d + 4 * hkv * d + tok), "flops": 4 * sum(lens) * hq * d}
    t = case["t"]
    if w == "prompt":
        return {"bytes": case["n"] * t * (4 * hq * d + 4 * hkv * d + tok), "flops": 4 * case["n"] * _causal_pairs(t) * hq * d}
    p = case["prefix"]
    return {"bytes": t * (4 * hq * d + 4 * hkv * d + tok) + p * tok + (p + t) * 4 * hkv * d, "flops": 4 * _causal_pairs(t, p) * hq * d}


def tolerance(case: dict):
    """About four times what the outputs were measured to be off by against the same mathematics in 64 bits."""
    w = case["work"]
    if w == "tensor":
        return "exact"
    if w in ("step", "hoststep"):
        # one rounding of the output to bf16 is 1.7e-3; over a quantised cache the softmax weights are fp16 operands, whose small
        # values cost more as the context grows (2.9e-3 at 16384 tokens, 7.6e-3 at 60000)
        if case["kind"] == "bf16":
            return {"rel": 0.007}
        return {"rel": 0.012 if case["hi"] <= 16384 else 0.03}
    if w in ("prompt", "chunk"):
        return {"rel": 0.009}  # 2.0e-3 to 2.3e-3
    if w == "qprompt":
        # 3.1e-3 (bf16 operands of the chunked rule; single values up to 0.4 of the rms); a key rounded to the other bf16 neighbour
        # after its norm changes its code: 1.4e-3 of the codes
        return {"rel": 0.0125, "max": 0.99, "differ": 0.0055}
    # 2.9e-3; of the cache's codes only the new tokens' can differ (4e-3 of one token's in 1024 or more)
    return {"rel": 0.012, "differ": 2e-5}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
NF4_VALUES = [-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334, -0.09105003625154495,
              0.0, 0.07958029955625534, 0.16093020141124725, 0.24611230945587158, 0.33791524171829224, 0.44070982933044434, 0.5626170039176941,
              0.7229568362236023, 1.0]


def _codebook(kind: int, dev) -> torch.Tensor:
    if kind == ffi.KV_INT8:
        return (torch.arange(256, device=dev, dtype=torch.float64) - 127.0) / 127.0
    if kind == ffi.KV_NF4:
        return torch.tensor(NF4_VALUES, device=dev, dtype=torch.float64)
    return torch.tensor([i / 16 for i in range(15)] + [1.0], device=dev, dtype=torch.float64)


def _rounded(x: torch.Tensor, kind: int, block: int, f16: bool):
    """(values, block maxima) of x as a cache of this kind holds them."""
    if kind == ffi.KV_BF16:
        return x.bfloat16().double(), None
    flat = x.double().flatten()
    n = flat.numel()
    flat = torch.nn.functional.pad(flat, (0, -n % block)).view(-1, block)
    top = flat.abs().amax(1, keepdim=True)
    top = top.half().double() if f16 else top
    book = _codebook(kind, x.device)
    at = torch.bucketize(flat / torch.where(top > 0, top, 1.0), (book[1:] + book[:-1]) / 2)
    return (book[at] * top).flatten()[:n].view(x.shape), top.flatten()


def _stored(cache: _Cache, s: int, length: int):
    """The first `length` tokens of sequence s as the cache's buffers hold them: (k, v) [length, heads, dim]."""
    view, page, kvs = cache.view, cache.view.page_tokens, []
    for i in (0, 1):
        def rows(t, table):
            slot = ((table[s] - t.data_ptr()) // (t.stride(0) * t.element_size()))[: (length + page - 1) // page]
            return t[slot].flatten(0, 1)[:length]
        codes = rows(cache.tensors[i], cache.tables[i])
        if cache.bf16:
            kvs.append(codes.contiguous().view(torch.bfloat16).double())
            continue
        if view.kind != ffi.KV_INT8:
            codes = torch.stack((codes >> 4, codes & 15), -1).flatten(-2)  # the even element sits in the high nibble
        top = rows(cache.tensors[2 + i], cache.tables[2 + i]).double().repeat_interleave(view.block, -1)
        kvs.append(_codebook(view.kind, codes.device)[codes.long()] * top)
    return kvs


def _rotated(x: torch.Tensor, sin, cos, pos, rotary: int) -> torch.Tensor:
    """Half-split rotation of x [rows, heads, dim]."""
    x = x.double()
    if sin is None:
        return x
    h = rotary // 2
    s, c = sin.double()[pos.long()][:, None], cos.double()[pos.long()][:, None]
    a, b = x[..., :h], x[..., h:rotary]
    return torch.cat([a * c - b * s, a * s + b * c, x[..., rotary:]], -1)


def _attend(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor) -> torch.Tensor:
    """Causal attention of q [T, Hq, D] over k, v [L, Hkv, D], the queries at the last T positions."""
    (t, hq, d), (l, hkv) = q.shape, k.shape[:2]
    out = torch.empty(t, hq, d, device=q.device, dtype=torch.float64)
    rows = max(1, (1 << 28) // (l * (hq // hkv)))
    for h in range(hkv):
        kh, vh, heads = k[:, h].double(), v[:, h].double(), slice(h * (hq // hkv), (h + 1) * (hq // hkv))
        for a in range(0, t, rows):
            b = min(t, a + rows)
            seen = l - t + b
            s = q[a:b, heads].double().transpose(0, 1) @ kh[:seen].T / math.sqrt(d)
            late = torch.arange(seen, device=q.device) > (l - t + torch.arange(a, b, device=q.device))[:, None]
            out[a:b, heads] = (s.masked_fill_(late, -math.inf).softmax(-1) @ vh[:seen]).transpose(0, 1)
    return out


def _delta_layer(layer, x, z, a, b, conv_state, state, carried: bool):
    """One gated-DeltaNet layer between its projections: (y, conv state, recurrent state)."""
    (n, t, conv), f = x.shape, torch.nn.functional
    front = conv_state.double() if carried else torch.zeros_like(conv_state, dtype=torch.float64)
    frames = torch.cat([front.transpose(1, 2), x.double()], 1)
    w = layer.conv_weight.double()
    mixed = f.silu(sum(frames[:, i:i + t] * w[:, i] for i in range(TAPS)))
    unit = lambda u: u / u.norm(dim=-1, keepdim=True).clamp_min(1e-3)  # noqa: E731
    q, k = (unit(u.reshape(n, t, NK, HD)).repeat_interleave(NV // NK, 2) for u in (mixed[..., :NK * HD], mixed[..., NK * HD:2 * NK * HD]))
    q, v = q / math.sqrt(HD), mixed[..., 2 * NK * HD:].reshape(n, t, NV, HD)
    g = layer.neg_a_exp.double() * f.softplus(a.double() + layer.dt_bias.double())
    decay, beta = g.exp(), torch.sigmoid(b.double())
    s, out = (state.double().clone() if carried else torch.zeros_like(state, dtype=torch.float64)), torch.empty_like(v)
    for i in range(t):
        s *= decay[:, i, :, None, None]
        ki = k[:, i, :, None, :]
        s += ki.transpose(-1, -2) * ((v[:, i, :, None, :] - ki @ s) * beta[:, i, :, None, None])
        out[:, i] = (q[:, i, :, None, :] @ s)[:, :, 0]
    norm = out * torch.rsqrt(out.square().mean(-1, keepdim=True) + 1e-6)
    return norm * layer.norm_weight.double() * f.silu(z.double()), frames[:, t:].transpose(1, 2).contiguous(), s


def exact(case: dict, seed: int):
    """What `run` returns, worked out in 64 bits; None for caches (their codes and block maxima are roundings of the inputs)."""
    st, w = prepare(case, seed), case["work"]
    if w == "tensor":
        values, top = _rounded(st["x"], st["kind"], st["block"], case["f16"])
        return [None, top, values]
    if w in ("qstep", "qprompt"):
        b, t, attn = st["b"], st["t"], st["attn"]
        if t * b > 70000:
            return None  # the recurrence takes too long one token at a time
        layers = [_delta_layer(l, *g, st["has"]) for l, g in zip(st["layers"], st["gin"])]
        qp, kp, v, _, pos, _, lens = st["ain"]

        def normed(x, weight):
            x = x.double()
            return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * (1.0 + weight.double())
        qg = qp.view(b * t, QHQ, 2 * QD)
        q = _rotated(normed(qg[..., :QD], attn.qw), attn.sin, attn.cos, pos, QROT).view(b, t, QHQ, QD)
        k = _rotated(normed(kp.view(b * t, QHKV, QD), attn.kw), attn.sin, attn.cos, pos, QROT).view(b, t, QHKV, QD)
        out = torch.empty(b, t, QHQ, QD, device=st["dev"], dtype=torch.float64)
        for s in range(b):
            ks, vs = k[s], v[s]
            if w == "qstep":
                old = _stored(st["cache"], s, int(lens[s]) - 1)
                ks, vs = (torch.cat([o, _rounded(x, ffi.KV_INT8, case["block"], case["f16"])[0]]) for o, x in zip(old, (ks, vs)))
            out[s] = _attend(q[s], ks, vs)
        out *= torch.sigmoid(qg[..., QD:].double().view(b, t, QHQ, QD))
        return [l[0] for l in layers] + [out] + [s for l in layers for s in l[1:]] + [None] * len(st["cache"].tensors)
    if w == "chunk":
        rnd, p, t, hkv, d = _Gen(seed), case["prefix"], case["t"], case["hkv"], case["d"]
        old = [rnd.b(1, p, hkv, d) for _ in range(2)]
        k, v = (_rounded(torch.cat([o, st[x]], 1), KINDS[case["kind"]], case["block"], case["f16"])[0] for o, x in zip(old, "kv"))
        return [_attend(st["q"][0], k[0], v[0])[None], k, v]
    cache, hkv, d, n = st["cache"], case["hkv"], case["d"], case["n"]
    none = [None] * len(cache.tensors)
    if w == "prompt":
        t = st["t"]
        q, k = (_rotated(st[x], st["sin"], st["cos"], st["pos"], st["rotary"]).view(n, t, -1, d) for x in "qk")
        return [torch.stack([_attend(q[s], k[s], st["v"][s]) for s in range(n)])] + none
    lens = st["lens"]
    q, k, v = (getattr(st["step"], x + "_host").to(lens.device) for x in "qkv") if w == "hoststep" else (st["q"], st["k"], st["v"])
    if w == "step":
        q = _rotated(q, st["sin"], st["cos"], lens - 1, st["rotary"])
    k = _rotated(k.reshape(n, hkv, d), st["sin"], st["cos"], lens - 1, st["rotary"])
    out = []
    for s in range(n):
        old, new = _stored(cache, s, int(lens[s]) - 1), (k[s:s + 1], v.reshape(n, 1, hkv, d)[s])
        ks, vs = (torch.cat([o, _rounded(x, KINDS[case["kind"]], case["block"], case["f16"])[0]]) for o, x in zip(old, new))
        out.append(_attend(q[s:s + 1], ks, vs))
    return [torch.cat(out)] + none
