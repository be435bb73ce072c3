"""GPU parity of the tcgen05 prompt-attention kernel (csrc/attention_prefill_umma.cu) at the sizes where its tiling can go wrong, against a float64 restatement
in torch.  Tolerance: P and the output are rounded to 16 bits, 2^-9 relative each for bf16 (2^-12 for f16), rounding errors of the terms of one output add up
in quadrature: relative Frobenius below 2^-8 (2^-11)."""
import numpy as np
import pytest
import torch

import candle_vllm_b200 as pkg
from candle_vllm_b200 import seq_ops
from tests.gpu_util import DEV

pytestmark = pytest.mark.gpu


def _reference(q, kc, vc, tables, qlens, klens, scale, window):
    out, at = [], 0
    for i, (n, k) in enumerate(zip(qlens, klens)):
        ids = torch.as_tensor(tables[i][: -(-k // 64)], device=q.device)
        keys, values = kc[ids].flatten(0, 1)[:k].double(), vc[ids].flatten(0, 1)[:k].double()
        g = q.shape[1] // keys.shape[1]
        keys, values = keys.repeat_interleave(g, 1), values.repeat_interleave(g, 1)
        s = torch.einsum("qhd,khd->hqk", q[at:at + n].double(), keys) * scale
        pos, key = torch.arange(k - n, k, device=q.device)[:, None], torch.arange(k, device=q.device)[None]
        hidden = key > pos if not window else (key > pos) | (key <= pos - window)
        out.append(torch.einsum("hqk,khd->qhd", torch.softmax(s.masked_fill(hidden, -np.inf), 2), values))
        at += n
    return torch.cat(out)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,kvh,qlens,cached,window,loud", [
    (4, 4, [1, 127, 128, 129, 257], [0, 1, 127, 128, 200], None, 1.0),      # one head per tile: 128 / 256 token tiles and one either side
    (8, 4, [63, 64, 65, 128], [64, 63, 0, 129], None, 1.0),                 # two heads per tile
    (32, 8, [1, 31, 32, 33, 63, 64, 65], [0, 700, 64, 31, 65, 64, 190], None, 1.0),   # four
    (24, 4, [70, 5], [10, 300], None, 1.0),                                 # groups of six: two heads share a tile
    (7, 1, [150], [77], None, 1.0),                                         # an odd group
    (32, 1, [9, 4, 3], [500, 0, 61], None, 1.0),                            # four tokens per tile
    (8, 2, [300, 40], [100, 250], 96, 1.0),                                 # window: starts inside the second page of a key tile
    (8, 2, [130], [400], 1, 1.0),                                           # a window of the token itself
    (8, 2, [200], [900], None, 6.0),                                        # loud scores: the running maximum moves by more than the slack, many times
])
def test_tiles_heads_and_edges(dtype, H, kvh, qlens, cached, window, loud):
    g = torch.Generator(device=DEV)
    g.manual_seed(H * 1000 + len(qlens))
    klens = [a + b for a, b in zip(qlens, cached)]
    used = [-(-k // 64) for k in klens]
    pool = sum(used) + 1
    perm = np.random.default_rng(H).permutation(pool)
    tables, at = [], 0
    for n in used:
        tables.append([int(x) for x in perm[at:at + n]])
        at += n
    mk = lambda *shape: torch.randn(shape, generator=g, device=DEV).to(dtype)
    q, k, v = mk(sum(qlens), H, 128) * loud, mk(sum(qlens), kvh, 128), mk(sum(qlens), kvh, 128)
    kc, vc = torch.full((pool, 64, kvh, 128), float("nan"), dtype=dtype, device=DEV), torch.full((pool, 64, kvh, 128), float("nan"), dtype=dtype, device=DEV)
    for i, c in enumerate(cached):                  # only what a context holds is written: everything else of the pool is NaN
        for j in range(-(-c // 64)):
            w = min(64, c - j * 64)
            kc[tables[i][j], :w], vc[tables[i][j], :w] = mk(w, kvh, 128), mk(w, kvh, 128)
    prep = pkg.prepare_prompt([list(range(n)) for n in klens], tables, 64, cached, chunk_size=max(qlens))
    _, _, meta = pkg.inputs.to_device(prep)
    out = pkg.PagedAttention(H, 128, 128 ** -0.5, kvh, sliding_window=window).forward(q, k, v, None, kc, vc, meta)
    ref = _reference(q, kc, vc, tables, qlens, klens, 128 ** -0.5, window)
    assert torch.isfinite(out).all()
    err = float((out.double() - ref).norm() / ref.norm())
    assert err < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11), err


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,kvh,qlens,cached,window,bad", [
    (4, 4, [200], [0], None, [(0, 1, "inf"), (0, 30, "nan"), (0, 127, "-inf"), (0, 128, "inf"), (0, 199, "nan")]),      # one head per tile: rows far before the values
    (8, 2, [130, 40], [300, 70], None, [(0, 17, "inf"), (0, 299, "nan"), (0, 301, "inf"), (0, 420, "-inf"), (1, 69, "nan"), (1, 100, "inf")]),
    (8, 2, [300], [500], 96, [(0, 0, "nan"), (0, 410, "inf"), (0, 480, "nan"), (0, 600, "-inf"), (0, 799, "inf")]),     # and behind a window's edge
    (32, 8, [1, 40], [700, 0], None, [(0, 700, "inf"), (1, 39, "nan")]),
    (8, 2, [200], [2900], None, [(0, 3, "inf"), (0, 100, "-inf"), (0, 2000, "nan"), (0, 3050, "inf")]),              # among the weights in two parts, seen by all
])
def test_values_that_are_not_finite_reach_the_rows_that_see_them_alone(dtype, H, kvh, qlens, cached, window, bad):
    g = torch.Generator(device=DEV)
    g.manual_seed(H + len(bad))
    klens = [a + b for a, b in zip(qlens, cached)]
    tables, at = [], 0
    for n in klens:
        tables.append(list(range(at, at - (-n // 64))))
        at += -(-n // 64)
    mk = lambda *shape: torch.randn(shape, generator=g, device=DEV).to(dtype)
    q, k, v = mk(sum(qlens), H, 128), mk(sum(qlens), kvh, 128), mk(sum(qlens), kvh, 128)
    kc, vc = mk(at, 64, kvh, 128), mk(at, 64, kvh, 128)
    first = np.cumsum([0] + qlens)
    clean = vc.clone()
    for i in range(len(qlens)):                    # what the call will write, so that the reference can start from it
        p = torch.arange(cached[i], klens[i], device=DEV)
        clean[torch.tensor(tables[i], device=DEV)[p // 64], p % 64] = v[first[i]:first[i + 1]]
    spoiled = clean.clone()
    for j, (i, pos, what) in enumerate(bad):
        group, dim = j % kvh, (37 * j + 5) % 128
        spoiled[tables[i][pos // 64], pos % 64, group, dim] = float(what)
        clean[tables[i][pos // 64], pos % 64, group, dim] = 0
    for i in range(len(qlens)):
        p = torch.arange(cached[i], klens[i], device=DEV)
        v[first[i]:first[i + 1]] = spoiled[torch.tensor(tables[i], device=DEV)[p // 64], p % 64]
    prep = pkg.prepare_prompt([list(range(n)) for n in klens], tables, 64, cached, chunk_size=max(qlens))
    _, _, meta = pkg.inputs.to_device(prep)
    vc.copy_(spoiled)
    out = pkg.PagedAttention(H, 128, 128 ** -0.5, kvh, sliding_window=window).forward(q, k, v, None, kc, vc, meta)
    ref = _reference(q, kc, clean, tables, qlens, klens, 128 ** -0.5, window)
    for j, (i, pos, what) in enumerate(bad):
        group, dim = j % kvh, (37 * j + 5) % 128
        rows = torch.arange(cached[i], klens[i], device=DEV)
        sees = (rows >= pos) & ((rows < pos + window) if window else torch.ones_like(rows, dtype=torch.bool))
        heads = slice(group * (H // kvh), (group + 1) * (H // kvh))
        ref[first[i]:first[i + 1], heads, dim] += torch.where(sees, float(what), 0.0)[:, None]
    finite = torch.isfinite(ref)
    assert torch.equal(torch.isfinite(out), finite)
    assert torch.equal(torch.isnan(out), torch.isnan(ref)) and torch.equal(out[torch.isinf(ref)].double(), ref[torch.isinf(ref)])
    err = float((out.double() - ref)[finite].norm() / ref[finite].norm())
    assert err < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11), err


@pytest.mark.parametrize("H,kvh,qlens,klens", [(4, 4, [600], [100]), (8, 2, [300, 40], [20, 64]), (4, 4, [300], [300])])
def test_rows_before_a_context_that_is_too_short_are_zero(H, kvh, qlens, klens):
    """more rows than keys: the mask is aligned at the end, so the first rows see nothing"""
    g = torch.Generator(device=DEV)
    g.manual_seed(sum(qlens))
    used = [-(-k // 64) for k in klens]
    tables = [list(range(sum(used[:i]), sum(used[:i + 1]))) for i in range(len(used))]
    mk = lambda *shape: torch.randn(shape, generator=g, device=DEV).to(torch.bfloat16)
    q, kc, vc = mk(sum(qlens), H, 128), mk(sum(used), 64, kvh, 128), mk(sum(used), 64, kvh, 128)
    k, v = mk(sum(qlens), kvh, 128), mk(sum(qlens), kvh, 128)
    meta = pkg.InputMetadata(is_prefill=True, slot_mapping=torch.full((sum(qlens),), -1, dtype=torch.int64, device=DEV),
                             block_tables=torch.tensor([t + [0] * (max(used) - len(t)) for t in tables], dtype=torch.int32, device=DEV), max_context_len=max(klens))
    on = lambda a: torch.tensor(np.cumsum([0] + a), dtype=torch.int32, device=DEV)
    meta.cu_seqlens_q, meta.cu_seqlens_k, meta.max_seqlen_q, meta.max_seqlen_k = on(qlens), on(klens), max(qlens), max(klens)
    out = pkg.PagedAttention(H, 128, 128 ** -0.5, kvh).forward(q, k, v, None, kc, vc, meta)
    row = 0
    for n, c, t in zip(qlens, klens, tables):
        blind = max(n - c, 0)
        assert not out[row:row + blind].any()
        ref = _reference(q[row + blind:row + n], kc, vc, [t], [n - blind], [c], 128 ** -0.5, None)
        assert float((out[row + blind:row + n].double() - ref).norm() / ref.norm()) < 2.0 ** -8
        row += n


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("new,cached,loud", [(700, 0, 1.0), (300, 1500, 1.0), (200, 5000, 1.0), (700, 1500, 3.0), (200, 5000, 3.0), (40, 0, 1.0)])
def test_no_less_precise_than_the_kernel_on_mma_sync(dtype, new, cached, loud):
    """Both round P to 16 bits once (mma.sync: against a maximum that is up to date every 32 keys).  A query that does not start on 16 bytes takes the mma.sync kernel, so
    both run on the same values.  Margin: 0.5 %, the spread of the ratio between draws of this size."""
    g = torch.Generator(device=DEV)
    g.manual_seed(new + cached)
    H, kvh, klen = 8, 2, new + cached
    used = -(-klen // 64)
    mk = lambda *shape: torch.randn(shape, generator=g, device=DEV).to(dtype)
    q, k, v = mk(new, H, 128) * loud, mk(new, kvh, 128), mk(new, kvh, 128)
    kc, vc = mk(used, 64, kvh, 128), mk(used, 64, kvh, 128)
    prep = pkg.prepare_prompt([list(range(klen))], [list(range(used))], 64, [cached], chunk_size=new)
    _, _, meta = pkg.inputs.to_device(prep)
    buf = torch.empty(q.numel() + 8, dtype=dtype, device=DEV)
    off = buf[4:4 + q.numel()].view(q.shape)
    off.copy_(q)
    assert q.data_ptr() % 16 == 0 and off.data_ptr() % 16 == 8
    op = pkg.PagedAttention(H, 128, 128 ** -0.5, kvh)
    errs = []
    for x in (off, q):
        out = op.forward(x, k, v, None, kc, vc, meta)
        ref = _reference(q, kc, vc, [list(range(used))], [new], [klen], 128 ** -0.5, None)
        errs.append(float((out.double() - ref).norm() / ref.norm()))
    assert errs[1] <= 1.005 * errs[0], errs


@pytest.mark.parametrize("H,kvh,qlens,cached,chunk,sink", [
    (8, 2, [257], [127], 128, False),              # a chunk border at the edge of a key tile, inside a query tile
    (8, 2, [300, 33], [190, 64], 192, True),       # chunks that are no multiple of a key tile, with a sink
    (4, 4, [129], [0], 64, True),
    (8, 2, [200, 1], [900, 700], 0, True),         # a sink over many key tiles
])
def test_chunks_and_sinks_at_tile_edges(H, kvh, qlens, cached, chunk, sink):
    g = torch.Generator(device=DEV)
    g.manual_seed(H + chunk)
    klens = [a + b for a, b in zip(qlens, cached)]
    tables, at = [], 0
    for n in klens:
        tables.append(list(range(at, at - (-n // 64))))
        at += -(-n // 64)
    mk = lambda *shape: torch.randn(shape, generator=g, device=DEV).to(torch.bfloat16)
    q, kc, vc = mk(sum(qlens), H, 128), mk(at, 64, kvh, 128), mk(at, 64, kvh, 128)
    s = torch.randn(H, generator=g, device=DEV) * 2 if sink else None
    prep = pkg.inputs.prepare_step([dict(tokens=[0] * n, start=c, block_table=t, slot=i) for i, (n, c, t) in enumerate(zip(qlens, cached, tables))], 64)
    batch = seq_ops.StepBatch.from_host(prep, DEV)
    out = seq_ops.paged_attention_varlen_sink(q.reshape(-1, H * 128), kc, vc, batch, H, kvh, 128, 128, 64, 128 ** -0.5, chunk, 0, s, torch.bfloat16).view(-1, H, 128)
    ref, row = [], 0
    for n, k, t in zip(qlens, klens, tables):
        keys, values = (c[torch.tensor(t, device=DEV)].flatten(0, 1)[:k].double().repeat_interleave(H // kvh, 1) for c in (kc, vc))
        score = torch.einsum("qhd,khd->hqk", q[row:row + n].double(), keys) * 128 ** -0.5
        pos, key = torch.arange(k - n, k, device=DEV)[:, None], torch.arange(k, device=DEV)[None]
        hidden = (key > pos) | (key < pos // chunk * chunk) if chunk else key > pos
        score = score.masked_fill(hidden, -np.inf)
        if sink:
            score = torch.cat([score, s.double()[:, None, None].expand(-1, n, 1)], 2)
        ref.append(torch.einsum("hqk,khd->qhd", torch.softmax(score, 2)[..., :k], values))
        row += n
    ref = torch.cat(ref)
    err = float((out.double() - ref).norm() / ref.norm())
    assert torch.isfinite(out).all() and err < 2.0 ** -8, err
