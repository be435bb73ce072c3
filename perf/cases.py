"""What is timed when this package's speed is measured: the calls a serving program makes, over the sizes it meets.

Seven kinds of calls, each through the package's public entry points: a decode or a prompt step of paged attention (cache write
included), the feed-forward of a GGUF model, a dense linear, a block of routed GGUF experts, latent attention with its cache write, and a
whole decode step of the Llama engine.  ``listed()`` names twelve of them; ``draw()`` gives more of the same ranges.  Every tensor is made
from the seed on the device, ``exact()`` restates the arithmetic in 64 bits with torch alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import candle_vllm_b200 as b200
from candle_vllm_b200 import mla

DEVICE = "cuda"
BLOCK = 64                                   # tokens per cache block, the serving default
TYPES = {"bf16": torch.bfloat16, "f16": torch.float16}
GGML = {"q4k": b200.GgmlType.Q4_K, "q6k": b200.GgmlType.Q6_K}
LATENT, ROPE = 512, 64                       # latent attention: compressed width, rotated width


# ---------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one chat request decoding alone: launches and latency are all there is
        dict(name="attn_decode_one", kind="attn_decode", batch=1, ctx=700, spread=0.0, heads=32, kv_heads=8, dtype="bf16", kv="same"),
        # a full batch of an 8B model, 4k prompts of unequal length: the cache is read at memory speed
        dict(name="attn_decode_batch", kind="attn_decode", batch=32, ctx=4608, spread=0.3, heads=32, kv_heads=8, dtype="bf16", kv="same"),
        # three requests' prompt portions on cached prefixes, lengths as they come
        dict(name="attn_prompt_ragged", kind="attn_prompt", seqs=3, new=701, prefix=1500, spread=0.6, heads=32, kv_heads=8, dtype="bf16"),
        # one prompt portion of the largest size the scheduler cuts
        dict(name="attn_prompt_long", kind="attn_prompt", seqs=1, new=8192, prefix=0, spread=0.0, heads=32, kv_heads=8, dtype="bf16"),
        # feed-forward of an 8B GGUF model, 32 requests decoding
        dict(name="mlp_decode", kind="mlp", m=32, hidden=4096, ffn=14336, ggml="q4k"),
        # the same with the wider quantisation while one short prompt is read
        dict(name="mlp_prompt", kind="mlp", m=203, hidden=4096, ffn=14336, ggml="q6k"),
        # a projection with bias for a short prompt
        dict(name="linear_short", kind="linear", m=100, n=4096, k=4096, dtype="bf16", bias=True),
        # the down projection for the largest prompt portion: the most arithmetic of all
        dict(name="linear_long", kind="linear", m=8192, n=4096, k=14336, dtype="bf16", bias=False),
        # routed experts, 16 requests decoding: a stream of the experts that were hit
        dict(name="moe_decode", kind="moe", tokens=16, experts=128, hidden=2048, inter=768, topk=8),
        # the same block while a prompt is read
        dict(name="moe_prompt", kind="moe", tokens=900, experts=128, hidden=2048, inter=768, topk=8),
        # latent attention, one rank's share of the heads, 32 requests decoding
        dict(name="mla_decode", kind="mla", batch=32, ctx=4096, spread=0.3, heads=16, dtype="bf16"),
        # a whole decode step: int4 weights, 8-bit cache
        dict(name="step_int4_kv8", kind="step", batch=32, ctx=4200, spread=0.2, layers=4, weights="int4", kv="fp8"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attn_decode", "attn_decode", "attn_prompt", "attn_prompt", "mlp", "mlp", "linear", "linear", "moe", "moe", "mla", "step"])
    dtype = rng.choice(["bf16", "bf16", "f16"])
    if kind == "attn_decode":
        heads, kv_heads = rng.choice([(32, 8), (32, 8), (32, 4), (16, 4), (8, 2), (16, 16)])
        batch = _log_int(rng, 1, 64)
        ctx = min(_log_int(rng, 16, 8192), 32 * 4608 // batch)
        return dict(kind=kind, batch=batch, ctx=ctx, spread=round(rng.uniform(0.0, 0.9), 2), heads=heads, kv_heads=kv_heads, dtype=dtype,
                    kv=rng.choice(["same", "same", "fp8"]))
    if kind == "attn_prompt":
        heads, kv_heads = rng.choice([(32, 8), (32, 8), (32, 4), (16, 4), (8, 2), (16, 16)])
        seqs = _log_int(rng, 1, 8)
        new = _log_int(rng, 16, 8192 // seqs)
        prefix = min(rng.choice([0, _log_int(rng, 64, 4096)]), 8192 - new)
        return dict(kind=kind, seqs=seqs, new=new, prefix=prefix, spread=round(rng.uniform(0.0, 0.9), 2), heads=heads, kv_heads=kv_heads, dtype=dtype)
    if kind == "mlp":
        hidden, ffn = rng.choice([(4096, 14336), (4096, 14336), (4096, 11008), (2048, 6144)])
        return dict(kind=kind, m=_log_int(rng, 1, 2048), hidden=hidden, ffn=ffn, ggml=rng.choice(["q4k", "q4k", "q6k"]) if ffn % 2048 == 0 else "q4k")
    if kind == "linear":
        n, k = rng.choice([(4096, 4096), (6144, 4096), (1024, 4096), (14336, 4096), (4096, 14336), (2048, 2048)])
        return dict(kind=kind, m=_log_int(rng, 1, 8192), n=n, k=k, dtype=dtype, bias=rng.choice([False, True]))
    if kind == "moe":
        experts, topk = rng.choice([(128, 8), (128, 8), (32, 4)])
        return dict(kind=kind, tokens=_log_int(rng, 1, 1024), experts=experts, hidden=2048, inter=768, topk=topk)
    if kind == "mla":
        batch = _log_int(rng, 1, 32)
        return dict(kind=kind, batch=batch, ctx=_log_int(rng, 64, 4608), spread=round(rng.uniform(0.0, 0.9), 2), heads=rng.choice([16, 16, 32, 128]), dtype=dtype)
    return dict(kind=kind, batch=_log_int(rng, 1, 32), ctx=_log_int(rng, 64, 4200), spread=round(rng.uniform(0.0, 0.6), 2), layers=4,
                weights=rng.choice(["q4k", "int4", "bf16"]), kv=rng.choice(["same", "fp8"]))


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _lengths(count, top, spread):
    """``count`` unequal lengths: the first is ``top``, the others lie up to ``spread`` below it."""
    return [max(1, round(top * (1.0 - spread * ((i * 0.6180339887) % 1.0)))) for i in range(count)]


class _Source:
    """Seeded tensors on the device."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEVICE)
        self.gen.manual_seed(int(seed))
        self.host = np.random.default_rng(int(seed))

    def normal(self, *shape, dtype=torch.float32, std=1.0):
        return (torch.randn(shape, generator=self.gen, device=DEVICE) * std).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.rand(shape, generator=self.gen, device=DEVICE) * (hi - lo) + lo

    def ints(self, hi, *shape, dtype=torch.int64):
        return torch.randint(0, hi, shape, generator=self.gen, device=DEVICE, dtype=dtype)

    def cache(self, *shape, kind):
        """cache contents: 16-bit values, or e4m3 bits"""
        if kind == "fp8":
            return self.normal(*shape).to(torch.float8_e4m3fn).view(torch.uint8)
        return self.normal(*shape, dtype=TYPES[kind])

    def tables(self, lens):
        """one row of scattered block ids per sequence, zero-padded, and the number of blocks in the pool"""
        used = [-(-n // BLOCK) for n in lens]
        pool = sum(used) + 3
        ids = self.host.permutation(pool)
        out, at = np.zeros((len(lens), max(used)), np.int32), 0
        for i, n in enumerate(used):
            out[i, :n] = ids[at:at + n]
            at += n
        return out, pool

    def ggml_blocks(self, ggml, rows, k):
        """valid random blocks, weights of zero mean and a standard deviation near 0.02"""
        count = rows * (k // 256)
        half = lambda v: v.to(torch.float16).view(torch.uint8).reshape(count, 2)
        if ggml == "q4k":
            b = torch.randint(0, 256, (count, 144), generator=self.gen, device=DEVICE, dtype=torch.uint8)
            b[:, 0:2] = half(self.uniform(count, lo=0.5, hi=2.0) * 2.0 ** -14)
            b[:, 2:4] = half(self.uniform(count, lo=0.5, hi=2.0) * 7.5 * 2.0 ** -14)
        else:
            b = torch.randint(0, 256, (count, 210), generator=self.gen, device=DEVICE, dtype=torch.uint8)
            b[:, 208:210] = half(self.uniform(count, lo=0.5, hi=2.0) * 2.0 ** -16)
        return b.reshape(-1)


def _slots(tables, seq, positions):
    return tables[seq, positions // BLOCK].astype(np.int64) * BLOCK + positions % BLOCK


def _on(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE)


def _attn_inputs(case, seed):
    s = _Source(seed)
    kvh, heads, dtype = case["kv_heads"], case["heads"], TYPES[case["dtype"]]
    kind = "fp8" if case.get("kv") == "fp8" else case["dtype"]
    if case["kind"] == "attn_decode":
        klen = _lengths(case["batch"], case["ctx"], case["spread"])
        qlen = [1] * len(klen)
    else:
        qlen = _lengths(case["seqs"], case["new"], case["spread"])
        before = _lengths(case["seqs"], case["prefix"], case["spread"]) if case["prefix"] else [0] * case["seqs"]
        klen = [a + b for a, b in zip(qlen, before)]
    tables, pool = s.tables(klen)
    rows = sum(qlen)
    slots = np.concatenate([_slots(tables, i, np.arange(k - q, k)) for i, (q, k) in enumerate(zip(qlen, klen))])
    return dict(qlen=qlen, klen=klen, tables=tables, slots=slots, k_cache=s.cache(pool, BLOCK, kvh, 128, kind=kind), v_cache=s.cache(pool, BLOCK, kvh, 128, kind=kind),
                q=s.normal(rows, heads, 128, dtype=dtype), k=s.normal(rows, kvh, 128, dtype=dtype), v=s.normal(rows, kvh, 128, dtype=dtype))


def _mlp_inputs(case, seed):
    s = _Source(seed)
    h, f = case["hidden"], case["ffn"]
    return dict(x=s.normal(case["m"], h), gate=s.ggml_blocks(case["ggml"], f, h), up=s.ggml_blocks(case["ggml"], f, h), down=s.ggml_blocks(case["ggml"], h, f))


def _linear_inputs(case, seed):
    s = _Source(seed)
    dtype = TYPES[case["dtype"]]
    return dict(x=s.normal(case["m"], case["k"], dtype=dtype), w=s.normal(case["n"], case["k"], dtype=dtype, std=0.02),
                bias=s.normal(case["n"], dtype=dtype) if case["bias"] else None)


def _moe_inputs(case, seed):
    s = _Source(seed)
    e, h, i = case["experts"], case["hidden"], case["inter"]
    return dict(x=s.normal(case["tokens"], h), router=s.normal(e, h, std=0.05), gate=s.ggml_blocks("q4k", e * i, h), up=s.ggml_blocks("q4k", e * i, h),
                down=s.ggml_blocks("q4k", e * h, i))


def _mla_inputs(case, seed):
    s = _Source(seed)
    dtype, heads = TYPES[case["dtype"]], case["heads"]
    klen = _lengths(case["batch"], case["ctx"], case["spread"])
    tables, pool = s.tables(klen)
    slots = np.array([_slots(tables, i, np.array([n - 1]))[0] for i, n in enumerate(klen)])
    return dict(klen=klen, tables=tables, slots=slots, ckv=s.normal(pool, BLOCK, 1, LATENT, dtype=dtype), kpe=s.normal(pool, BLOCK, 1, ROPE, dtype=dtype),
                q=s.normal(case["batch"], heads, LATENT, dtype=dtype, std=0.3), q_pe=s.normal(case["batch"], heads, ROPE, dtype=dtype, std=0.3),
                new_ckv=s.normal(case["batch"], LATENT, dtype=dtype), new_kpe=s.normal(case["batch"], ROPE, dtype=dtype))


# the engine's model: an 8B decoder's layers under a small vocabulary
_STEP = dict(hidden=4096, num_heads=32, num_kv_heads=8, head_dim=128, ffn=14336, vocab=16384)
_STEP_LINEARS = dict(wq=(4096, 4096), wk=(1024, 4096), wv=(1024, 4096), wo=(4096, 4096), w1=(14336, 4096), w2=(4096, 14336), w3=(14336, 4096))
_GROUP = 128                                 # int4: weights per scale


def _step_inputs(case, seed):
    s = _Source(seed)
    klen = _lengths(case["batch"], case["ctx"], case["spread"])
    tables, pool = s.tables(klen)

    def weight(n, k):
        if case["weights"] == "q4k":
            return s.ggml_blocks("q4k", n, k)
        if case["weights"] == "bf16":
            return s.normal(n, k, dtype=torch.bfloat16, std=0.02)
        return torch.randint(-2 ** 31, 2 ** 31, (k // 8, n), generator=s.gen, device=DEVICE, dtype=torch.int64).to(torch.int32), \
            s.uniform(k // _GROUP, n, lo=0.002, hi=0.006).to(torch.float16)

    kind = "fp8" if case["kv"] == "fp8" else "bf16"
    layers = []
    for _ in range(case["layers"]):
        layer = {name: weight(n, k) for name, (n, k) in _STEP_LINEARS.items()}
        layer.update(attn_norm=s.uniform(4096, lo=0.5, hi=1.5), ffn_norm=s.uniform(4096, lo=0.5, hi=1.5),
                     kv=(s.cache(pool, BLOCK, 8, 128, kind=kind), s.cache(pool, BLOCK, 8, 128, kind=kind)))
        layers.append(layer)
    return dict(klen=klen, tables=tables, layers=layers, tokens=s.host.integers(0, _STEP["vocab"], case["batch"]), embedding=s.normal(_STEP["vocab"], 4096),
                norm=s.uniform(4096, lo=0.5, hi=1.5),
                output=s.normal(_STEP["vocab"], 4096, dtype=torch.bfloat16, std=0.02) if case["weights"] == "bf16" else s.ggml_blocks("q6k", _STEP["vocab"], 4096))


# ---------------------------------------------------------------------------------------------------------------------
# what a program holds before the call, and the call
# ---------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("attn_decode", "attn_prompt"):
        d = _attn_inputs(case, seed)
        op = b200.PagedAttention(case["heads"], 128, 128 ** -0.5, case["kv_heads"], fp8_kvcache=case.get("kv") == "fp8")
        meta = b200.InputMetadata(is_prefill=kind == "attn_prompt", slot_mapping=_on(d["slots"]), block_tables=_on(d["tables"]), max_context_len=max(d["klen"]))
        if meta.is_prefill:
            meta.cu_seqlens_q = _on(np.cumsum([0] + d["qlen"]).astype(np.int32))
            meta.cu_seqlens_k = _on(np.cumsum([0] + d["klen"]).astype(np.int32))
            meta.max_seqlen_q, meta.max_seqlen_k = max(d["qlen"]), max(d["klen"])
        else:
            meta.context_lens = _on(np.array(d["klen"], np.int32))
        return dict(kind=kind, op=op, meta=meta, **{n: d[n] for n in ("q", "k", "v", "k_cache", "v_cache")})
    if kind == "mlp":
        d = _mlp_inputs(case, seed)
        h, f, t = case["hidden"], case["ffn"], GGML[case["ggml"]]
        linear = lambda data, n, k: b200.QMatMul.from_arc(b200.QTensor(data, t, (n, k)))
        return dict(kind=kind, x=d["x"], gate=linear(d["gate"], f, h), up=linear(d["up"], f, h), down=linear(d["down"], h, f))
    if kind == "linear":
        d = _linear_inputs(case, seed)
        return dict(kind=kind, x=d["x"], op=b200.Linear(d["w"], d["bias"]))
    if kind == "moe":
        d = _moe_inputs(case, seed)
        t = b200.GgmlType.Q4_K
        op = b200.FusedMoe(d["router"], d["gate"], d["up"], d["down"], (t, t, t), case["experts"], case["hidden"], case["inter"], case["topk"])
        return dict(kind=kind, x=d["x"], op=op, prompt=case["tokens"] > 64)
    if kind == "mla":
        d = _mla_inputs(case, seed)
        return dict(kind=kind, tables=_on(d["tables"]), lens=_on(np.array(d["klen"], np.int32)), slots=_on(d["slots"]), scale=(128 + ROPE) ** -0.5,
                    **{n: d[n] for n in ("q", "q_pe", "ckv", "kpe", "new_ckv", "new_kpe")})
    d = _step_inputs(case, seed)
    cfg = b200.LlamaConfig(num_layers=case["layers"], max_pos=8192, block_size=BLOCK, max_num_seqs=32, max_blocks_per_seq=128, **_STEP)

    def held(w, n, k):
        if case["weights"] == "bf16":
            return w
        if case["weights"] == "q4k":
            return b200.QTensor(w, b200.GgmlType.Q4_K, (n, k))
        return b200.MarlinWeight(b200.marlin_weight_repack(w[0], 4, False), b200.marlin_permute_scales(w[1], k, n, _GROUP), _GROUP)

    layers = [dict(attn_norm=l["attn_norm"], ffn_norm=l["ffn_norm"], **{name: held(l[name], n, k) for name, (n, k) in _STEP_LINEARS.items()}) for l in d["layers"]]
    output = d["output"] if case["weights"] == "bf16" else b200.QTensor(d["output"], b200.GgmlType.Q6_K, (_STEP["vocab"], 4096))
    model = b200.GGUFLLaMa(cfg, dict(tok_embeddings=d["embedding"], norm=d["norm"], output=output, layers=layers), [l["kv"] for l in d["layers"]],
                           kv_dtype=b200.DType.FP8_E4M3 if case["kv"] == "fp8" else b200.DType.BF16)
    return dict(kind=kind, model=model, prep=b200.prepare_decode(d["klen"], d["tokens"], d["tables"].tolist(), BLOCK))


def run(state):
    s, kind = state, state["kind"]
    if kind in ("attn_decode", "attn_prompt"):
        return dict(out=s["op"].forward(s["q"], s["k"], s["v"], None, s["k_cache"], s["v_cache"], s["meta"]), k_cache=s["k_cache"], v_cache=s["v_cache"])
    if kind == "mlp":
        return s["down"].forward(b200.silu_mul(s["gate"].forward(s["x"]), s["up"].forward(s["x"])))
    if kind == "linear":
        return s["op"].forward(s["x"])
    if kind == "moe":
        return s["op"].forward(s["x"], s["prompt"])
    if kind == "mla":
        mla.concat_and_cache_mla(s["new_ckv"], s["new_kpe"], s["ckv"], s["kpe"], s["slots"])
        out = mla.mla_paged_decode(s["q"], s["q_pe"], s["ckv"], s["kpe"], s["tables"], s["lens"], s["scale"])
        return dict(out=out, ckv=s["ckv"], kpe=s["kpe"])
    return s["model"].decode(s["prep"], want_logits=True)[1]


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
_GGML_BYTES = {"q4k": 144 / 256, "q6k": 210 / 256}


def work(case):
    kind = case["kind"]
    if kind in ("attn_decode", "attn_prompt"):
        heads, kvh = case["heads"], case["kv_heads"]
        each = 1 if case.get("kv") == "fp8" else 2
        if kind == "attn_decode":
            klen = _lengths(case["batch"], case["ctx"], case["spread"])
            qlen = [1] * len(klen)
        else:
            qlen = _lengths(case["seqs"], case["new"], case["spread"])
            before = _lengths(case["seqs"], case["prefix"], case["spread"]) if case["prefix"] else [0] * case["seqs"]
            klen = [a + b for a, b in zip(qlen, before)]
        pairs = sum(q * (k - q) + q * (q + 1) // 2 for q, k in zip(qlen, klen))
        rows = sum(qlen)
        return dict(bytes=sum(klen) * kvh * 256 * each + rows * (2 * heads + 2 * kvh) * 256 + rows * kvh * 256 * each, flops=4.0 * pairs * heads * 128)
    if kind == "mlp":
        weights = 3 * case["hidden"] * case["ffn"]
        return dict(bytes=weights * _GGML_BYTES[case["ggml"]] + case["m"] * case["hidden"] * 8, flops=2.0 * case["m"] * weights)
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return dict(bytes=2 * (m * k + n * k + m * n), flops=2.0 * m * n * k)
    if kind == "moe":
        t, e, k = case["tokens"], case["experts"], case["topk"]
        expert = 3 * case["hidden"] * case["inter"]
        hit = e * (1.0 - (1.0 - k / e) ** t)
        return dict(bytes=hit * expert * _GGML_BYTES["q4k"] + e * case["hidden"] * 4 + t * case["hidden"] * 8, flops=2.0 * t * k * expert + 2.0 * t * e * case["hidden"])
    if kind == "mla":
        total = sum(_lengths(case["batch"], case["ctx"], case["spread"]))
        return dict(bytes=2 * total * (LATENT + ROPE) + 2 * case["batch"] * case["heads"] * (2 * LATENT + ROPE), flops=2.0 * total * case["heads"] * (2 * LATENT + ROPE))
    total = sum(_lengths(case["batch"], case["ctx"], case["spread"]))
    weights = sum(n * k for n, k in _STEP_LINEARS.values()) * case["layers"]
    head = _STEP["vocab"] * 4096
    per = {"q4k": _GGML_BYTES["q4k"], "int4": 0.5 + 2 / _GROUP, "bf16": 2.0}[case["weights"]]
    return dict(bytes=weights * per + head * (2.0 if case["weights"] == "bf16" else _GGML_BYTES["q6k"]) + case["layers"] * total * 2048 * (1 if case["kv"] == "fp8" else 2)
                + case["batch"] * (_STEP["vocab"] + 4096) * 4,
                flops=2.0 * case["batch"] * (weights + head) + 4.0 * total * 4096 * case["layers"])


def tolerance(case):
    """About four times what the call is off the 64-bit result, which is what its data types give: 16-bit results of 16-bit operands (attention:
    probabilities rounded too), f32 results of products with f16 operands; through a whole step these add up layer by layer."""
    kind = case["kind"]
    if kind in ("attn_decode", "attn_prompt", "mla"):
        return dict(rel=1e-2 if case["dtype"] == "bf16" else 1.2e-3, max=0.2)
    if kind == "linear":
        return dict(rel=7e-3 if case["dtype"] == "bf16" else 1e-3, max=0.05)
    if kind in ("mlp", "moe"):
        return dict(rel=2.5e-3, max=0.05)
    return dict(rel=2e-2 if case["weights"] == "bf16" else 1e-2, max=0.3)


# ---------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def _dequantised(ggml, blocks, rows, k):
    """GGML blocks -> f64 [rows, k]"""
    if ggml == "q4k":
        b = blocks.view(-1, 144)
        d, dmin = (b[:, o:o + 2].contiguous().view(torch.float16).double() for o in (0, 2))
        s = b[:, 4:16].long()
        low, mid, high = s[:, 0:4], s[:, 4:8], s[:, 8:12]
        sc = torch.cat([low & 63, (high & 15) | (low >> 6 << 4)], 1)
        mn = torch.cat([mid & 63, (high >> 4) | (mid >> 6 << 4)], 1)
        q = b[:, 16:].view(-1, 4, 32)
        q = torch.stack([q & 15, q >> 4], 2).reshape(-1, 8, 32)
        return ((d * sc).unsqueeze(2) * q - (dmin * mn).unsqueeze(2)).reshape(rows, k)
    b = blocks.view(-1, 210)
    d = b[:, 208:210].contiguous().view(torch.float16).double()
    low, high = b[:, :128].view(-1, 2, 2, 32), b[:, 128:192].view(-1, 2, 1, 32)
    q = torch.cat([low & 15, low >> 4], 2).int() | (torch.cat([high, high >> 2, high >> 4, high >> 6], 2) & 3).int() << 4
    sc = b[:, 192:208].contiguous().view(torch.int8).double()
    return ((d * sc).unsqueeze(2) * (q.reshape(-1, 16, 16).double() - 32)).reshape(rows, k)


def _values(cache):
    return (cache.view(torch.float8_e4m3fn) if cache.dtype == torch.uint8 else cache).double()


def _written(cache, rows, slots):
    """the cache with ``rows`` at ``slots``, rounded as it stores them"""
    out = cache.clone()
    out.view(-1, *cache.shape[2:])[_on(slots)] = rows.to(torch.float8_e4m3fn).view(torch.uint8) if cache.dtype == torch.uint8 else rows.to(cache.dtype)
    return out


def _attention(q, keys, values, scale):
    """q f64 [n, H, dk] at the last n positions, keys [K, G, dk], values [K, G, dv] -> [n, H, dv]"""
    n, total, group = q.shape[0], keys.shape[0], q.shape[1] // keys.shape[1]
    out = torch.empty(n, q.shape[1], values.shape[2], dtype=torch.float64, device=q.device)
    hidden = torch.ones(n, total, dtype=torch.bool, device=q.device).triu_(total - n + 1)
    for h in range(q.shape[1]):
        s = (q[:, h] @ keys[:, h // group].T * scale).masked_fill_(hidden, -math.inf)
        out[:, h] = torch.softmax(s, 1) @ values[:, h // group]
    return out


def _paged(cache, table, length):
    used = -(-length // BLOCK)
    return _values(cache[_on(table[:used]).long()]).flatten(0, 1)[:length]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("attn_decode", "attn_prompt"):
        d = _attn_inputs(case, seed)
        kc, vc = _written(d["k_cache"], d["k"], d["slots"]), _written(d["v_cache"], d["v"], d["slots"])
        out, at = [], 0
        for i, (q, k) in enumerate(zip(d["qlen"], d["klen"])):
            out.append(_attention(d["q"][at:at + q].double(), _paged(kc, d["tables"][i], k), _paged(vc, d["tables"][i], k), 128 ** -0.5))
            at += q
        whole = kc.dtype != torch.uint8
        return dict(out=torch.cat(out), k_cache=kc if whole else None, v_cache=vc if whole else None)
    if kind == "mlp":
        d = _mlp_inputs(case, seed)
        h, f, x = case["hidden"], case["ffn"], d["x"].double()
        a = torch.nn.functional.silu(x @ _dequantised(case["ggml"], d["gate"], f, h).T) * (x @ _dequantised(case["ggml"], d["up"], f, h).T)
        return a @ _dequantised(case["ggml"], d["down"], h, f).T
    if kind == "linear":
        d = _linear_inputs(case, seed)
        y = d["x"].double() @ d["w"].double().T
        return y if d["bias"] is None else y + d["bias"].double()
    if kind == "moe":
        d = _moe_inputs(case, seed)
        e, h, i, x = case["experts"], case["hidden"], case["inter"], d["x"].double()
        p, ids = torch.softmax(x @ d["router"].double().T, 1).topk(case["topk"], 1)
        p = p / p.sum(1, keepdim=True)
        gate, up, down = (d[n].view(e, -1) for n in ("gate", "up", "down"))
        out = torch.zeros_like(x)
        for j in range(e):
            rows, slot = (ids == j).nonzero(as_tuple=True)
            if rows.numel():
                a = torch.nn.functional.silu(x[rows] @ _dequantised("q4k", gate[j], i, h).T) * (x[rows] @ _dequantised("q4k", up[j], i, h).T)
                out[rows] += p[rows, slot, None] * (a @ _dequantised("q4k", down[j], h, i).T)
        return out
    if kind == "mla":
        d = _mla_inputs(case, seed)
        ckv, kpe = _written(d["ckv"], d["new_ckv"].unsqueeze(1), d["slots"]), _written(d["kpe"], d["new_kpe"].unsqueeze(1), d["slots"])
        q, out = torch.cat([d["q"], d["q_pe"]], 2).double(), []
        for i, n in enumerate(d["klen"]):
            c, r = _paged(ckv, d["tables"][i], n), _paged(kpe, d["tables"][i], n)
            out.append(_attention(q[i:i + 1], torch.cat([c, r], 2), c, (128 + ROPE) ** -0.5))
        return dict(out=torch.cat(out), ckv=ckv, kpe=kpe)
    return _exact_step(case, seed)


def _exact_step(case, seed):
    d = _step_inputs(case, seed)

    def product(x, w, n, k):
        if case["weights"] == "q4k":
            return x @ _dequantised("q4k", w, n, k).T
        if case["weights"] == "bf16":
            return x @ w.double().T
        q = torch.stack([(w[0] >> (4 * j)) & 15 for j in range(8)], 1).reshape(k, n)
        return x @ ((q - 8).double() * w[1].double().repeat_interleave(_GROUP, 0))

    def norm(x, w):
        return x * torch.rsqrt(x.square().mean(1, keepdim=True) + 1e-5) * w.double()

    pos = torch.tensor(d["klen"], device=DEVICE).double() - 1
    angle = pos[:, None] * 500000.0 ** (-torch.arange(0, 128, 2, device=DEVICE).double() / 128)
    cos, sin = angle.cos().unsqueeze(1), angle.sin().unsqueeze(1)

    def turned(x):                               # neighbouring pairs, as the GGUF models store them
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).flatten(-2)

    slots = np.concatenate([_slots(d["tables"], i, np.array([n - 1])) for i, n in enumerate(d["klen"])])
    x = d["embedding"].double()[_on(d["tokens"])]
    rows = x.shape[0]
    for l in d["layers"]:
        p = lambda name, t: product(t, l[name], *_STEP_LINEARS[name])
        h = norm(x, l["attn_norm"])
        q, k, v = turned(p("wq", h).view(rows, 32, 128)), turned(p("wk", h).view(rows, 8, 128)), p("wv", h).view(rows, 8, 128)
        kc, vc = _written(l["kv"][0], k, slots), _written(l["kv"][1], v, slots)
        o = torch.cat([_attention(q[i:i + 1], _paged(kc, d["tables"][i], n), _paged(vc, d["tables"][i], n), 128 ** -0.5) for i, n in enumerate(d["klen"])])
        x = x + p("wo", o.flatten(1))
        h = norm(x, l["ffn_norm"])
        x = x + p("w2", torch.nn.functional.silu(p("w1", h)) * p("w3", h))
    x = norm(x, d["norm"])
    return x @ (d["output"].double() if case["weights"] == "bf16" else _dequantised("q6k", d["output"], _STEP["vocab"], 4096)).T
