"""Multi-head latent attention over the paged latent cache: mirror of the attention-rs MLA calls made by ``MlaAttention::forward``
(src/openai/models/layers/mla_attention.rs:479-552) over the C ABI (``concat_and_cache_mla``, ``mla_paged_attention``)."""
from __future__ import annotations

from typing import Optional

import torch

from ._lib import BackendError, calls, check, fail, require_device, typed
from .backend import _F, _I, _L, _P, _Z, _at, _cuda, _dt, _guard, _raw_stream


def concat_and_cache_mla(ckv: torch.Tensor, k_pe: torch.Tensor, ckv_cache: torch.Tensor, kpe_cache: torch.Tensor, slot_mapping: torch.Tensor) -> None:
    """ckv [T, R], k_pe [T, P] -> caches [nb, bs, 1, R] / [nb, bs, 1, P] at slot_mapping (i64; negative = pad)."""
    native = calls()
    if native:
        r = native.latent_cache(ckv, k_pe, ckv_cache, kpe_cache, slot_mapping)
        if r is not None:
            return fail("concat_and_cache_mla", r) if r else None
    for t, n in ((ckv, "ckv"), (k_pe, "k_pe"), (ckv_cache, "ckv_cache"), (kpe_cache, "kpe_cache"), (slot_mapping, "slot_mapping")):
        _cuda(t, n)
    require_device()
    if ckv.dtype != ckv_cache.dtype or k_pe.dtype != kpe_cache.dtype or ckv.dtype not in (torch.float16, torch.bfloat16):
        raise BackendError("concat_and_cache_mla: 16-bit tensors of the cache dtype expected")
    c, r, slots = ckv.contiguous(), k_pe.contiguous(), slot_mapping.contiguous()
    with _guard(ckv.device):
        typed("concat_and_cache_mla", None, _P, _P, _P, _P, _P, _I, _I, _I, _I, _L)(
            c.data_ptr(), r.data_ptr(), ckv_cache.data_ptr(), kpe_cache.data_ptr(), slots.data_ptr(), ckv.shape[0], ckv.shape[-1], k_pe.shape[-1], _dt(ckv),
            _raw_stream(ckv.device))
    check("concat_and_cache_mla")


def _mla(q_absorbed, q_pe, ckv_cache, kpe_cache, block_tables, context_lens, cu_seqlens_q, sm_scale):
    _cuda(q_absorbed, "q_absorbed"); require_device()
    rows, H, R = q_absorbed.shape
    P = q_pe.shape[-1]
    nb, bs = ckv_cache.shape[0], ckv_cache.shape[1]
    if q_absorbed.dtype != ckv_cache.dtype or q_absorbed.dtype not in (torch.float16, torch.bfloat16):
        raise BackendError("mla attention: q and the latent cache must share a 16-bit dtype")
    out = torch.empty((rows, H, R), dtype=q_absorbed.dtype, device=q_absorbed.device)
    B, W = block_tables.shape
    dev = q_absorbed.device
    need = typed("mla_paged_decode_workspace_bytes", _Z, _I, _I, _I, _I)(B, H, W, bs)
    ws = torch.empty(need, dtype=torch.uint8, device=dev)
    qa, qp = q_absorbed.contiguous(), q_pe.contiguous()
    tables, lens = block_tables.to(torch.int32).contiguous(), context_lens.to(torch.int32).contiguous()
    cu = None if cu_seqlens_q is None else cu_seqlens_q.to(torch.int32).contiguous()
    with _guard(dev):
        typed("mla_paged_attention", None, _P, _P, _P, _P, _P, _P, _P, _P, _I, _I, _I, _I, _I, _I, _I, _L, _F, _I, _P, _Z, _L)(
            out.data_ptr(), qa.data_ptr(), qp.data_ptr(), ckv_cache.data_ptr(), kpe_cache.data_ptr(), tables.data_ptr(), lens.data_ptr(), _at(cu), B, rows, H, R, P,
            bs, W, nb, sm_scale, _dt(q_absorbed), ws.data_ptr(), need, _raw_stream(dev))
    check("mla_paged_attention")
    return out


def mla_paged_decode(q_absorbed, q_pe, ckv_cache, kpe_cache, block_tables, context_lens, sm_scale: float) -> torch.Tensor:
    """attention_rs::mla::mla_paged_decode (mla_attention.rs:541-550): one query row per sequence -> [B, H, kv_lora_rank]."""
    native = calls()
    if native:
        r = native.latent_decode(q_absorbed, q_pe, ckv_cache, kpe_cache, block_tables, context_lens, sm_scale)
        if r is not None:
            return r if r.__class__ is not int else fail("mla_paged_attention", r)
    return _mla(q_absorbed, q_pe, ckv_cache, kpe_cache, block_tables, context_lens, None, sm_scale)


def mla_paged_prefill(q_absorbed, q_pe, ckv_cache, kpe_cache, block_tables, context_lens, cu_seqlens_q, sm_scale: float) -> torch.Tensor:
    """attention_rs::mla::mla_paged_prefill (mla_attention.rs:527-537): causal, rows = the last positions of each sequence's context."""
    return _mla(q_absorbed, q_pe, ckv_cache, kpe_cache, block_tables, context_lens, cu_seqlens_q, sm_scale)
