"""The merge of the decode kernel's chunk partials: a warp per head (head counts that are no multiple of four), chunk counts on either side of what is loaded ahead (8) and of what a warp's
lanes hold (32), chunks that the decode kernel has halved, outputs that start on an odd multiple of two bytes."""
import ctypes as C

import pytest
import torch

import candle_vllm_b200 as pkg

pytestmark = pytest.mark.gpu


def _reference(q, kc, vc, tables, lens, group):
    out = []
    for b, n in enumerate(lens):
        k = kc[tables[b, :-(-n // 64)].long()].flatten(0, 1)[:n].double().repeat_interleave(group, 1)
        v = vc[tables[b, :-(-n // 64)].long()].flatten(0, 1)[:n].double().repeat_interleave(group, 1)
        p = torch.softmax(torch.einsum("hd,khd->hk", q[b].double(), k) * 128 ** -0.5, 1)
        out.append(torch.einsum("hk,khd->hd", p, v))
    return torch.stack(out)


@pytest.mark.parametrize("heads,kv_heads", [(1, 1), (6, 3), (8, 2), (8, 1), (32, 8)])
@pytest.mark.parametrize("lens", [[1], [64 * 8], [64 * 8 + 1], [64 * 32, 3], [64 * 32 + 1], [64 * 70 + 5, 64, 700], [4600, 4664, 4300, 17] * 8])
@pytest.mark.parametrize("offset", [0, 1])
def test_merge(heads, kv_heads, lens, offset):
    gen = torch.Generator(device="cuda").manual_seed(len(lens) + heads)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    width = max(-(-n // 64) for n in lens)
    blocks = 300
    kc, vc, q = mk(blocks, 64, kv_heads, 128), mk(blocks, 64, kv_heads, 128), mk(len(lens), heads, 128)
    tables = torch.randint(0, blocks, (len(lens), width), generator=gen, device="cuda", dtype=torch.int32)
    ctx = torch.tensor(lens, dtype=torch.int32, device="cuda")
    held = torch.zeros(q.numel() + 8, dtype=torch.bfloat16, device="cuda")
    L = pkg.lib()
    ws = torch.zeros(int(L.paged_attention_decode_workspace_bytes(*map(C.c_int32, (len(lens), heads, 128, width, 64)))), dtype=torch.uint8, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())
    out = held[offset:offset + q.numel()].view_as(q)
    for _ in range(2):                                    # the work queue is left as it was found
        L.paged_attention_decode(p(out), p(q), p(kc), p(vc), p(tables), p(ctx), *map(C.c_int32, (len(lens), heads, kv_heads, 128, 64, width)), C.c_int64(blocks), C.c_float(128 ** -0.5),
                                 C.c_float(0), *map(C.c_int32, (0, 2, 2, 0, 2)), p(ws), C.c_size_t(ws.numel()), C.c_int64(torch.cuda.current_stream().cuda_stream))
        assert L.b200_last_error() == 0
    ref = _reference(q, kc, vc, tables, lens, heads // kv_heads)
    # weights and result rounded to bf16: 2^-9 / sqrt(3) each in the mean square
    assert float((out.double() - ref).norm() / ref.norm()) < 2.5e-3
    assert not held[:offset].any() and not held[offset + q.numel():].any()


@pytest.mark.parametrize("shift", [4, 8, 12, 2])
def test_workspace_may_start_on_any_word(shift):
    """the merge's 16-byte reads are aligned inside the workspace; one that starts inside a word is refused before anything is launched"""
    lens, heads, kv_heads, width = [700, 64 * 9 + 1], 8, 2, 11
    gen = torch.Generator(device="cuda").manual_seed(shift)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    kc, vc, q = mk(30, 64, kv_heads, 128), mk(30, 64, kv_heads, 128), mk(2, heads, 128)
    tables = torch.randint(0, 30, (2, width), generator=gen, device="cuda", dtype=torch.int32)
    ctx = torch.tensor(lens, dtype=torch.int32, device="cuda")
    L = pkg.lib()
    need = int(L.paged_attention_decode_workspace_bytes(*map(C.c_int32, (2, heads, 128, width, 64))))
    held = torch.zeros(need + 64, dtype=torch.uint8, device="cuda")
    held[shift + need:] = 7
    p = lambda t, by=0: C.c_void_p(t.data_ptr() + by)

    def call(by):
        out = torch.zeros_like(q)
        L.paged_attention_decode(p(out), p(q), p(kc), p(vc), p(tables), p(ctx), *map(C.c_int32, (2, heads, kv_heads, 128, 64, width)), C.c_int64(30), C.c_float(128 ** -0.5),
                                 C.c_float(0), *map(C.c_int32, (0, 2, 2, 0, 2)), p(held, by), C.c_size_t(need), C.c_int64(torch.cuda.current_stream().cuda_stream))
        return out, L.b200_last_error()

    if shift % 4:
        out, code = call(shift)
        assert code != 0 and b"workspace" in L.b200_last_error_message() and not out.any() and not held[:need].any()
        return
    outs = [call(shift), call(shift)]
    assert (held[shift + need:] == 7).all()
    held[:shift + need] = 0
    outs.append(call(0))
    assert all(code == 0 and torch.equal(out, outs[2][0]) for out, code in outs)
    ref = _reference(q, kc, vc, tables, lens, heads // kv_heads)
    assert float((outs[0][0].double() - ref).norm() / ref.norm()) < 2.5e-3


@pytest.mark.parametrize("lens,width", [([700, 100, 64], 128), ([1, 700, 2100], 128), ([3000], 47), ([4200, 64, 2048, 2049], 66)])
def test_merge_looks_at_written_partials_only(lens, width):
    """partials that the chunk size which decode kernel and merge settle for leaves out are not looked at; tables wider than the contexts, few and many chunks in one launch"""
    heads, kv_heads = 8, 2
    gen = torch.Generator(device="cuda").manual_seed(width)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    kc, vc, q = mk(80, 64, kv_heads, 128), mk(80, 64, kv_heads, 128), mk(len(lens), heads, 128)
    tables = torch.randint(0, 80, (len(lens), width), generator=gen, device="cuda", dtype=torch.int32)
    ctx = torch.tensor(lens, dtype=torch.int32, device="cuda")
    L = pkg.lib()
    need = int(L.paged_attention_decode_workspace_bytes(*map(C.c_int32, (len(lens), heads, 128, width, 64))))
    ws = torch.full((need,), 255, dtype=torch.uint8, device="cuda")                # NaN everywhere but in the header
    ws[:256] = 0
    out = torch.zeros_like(q)
    p = lambda t: C.c_void_p(t.data_ptr())
    L.paged_attention_decode(p(out), p(q), p(kc), p(vc), p(tables), p(ctx), *map(C.c_int32, (len(lens), heads, kv_heads, 128, 64, width)), C.c_int64(80), C.c_float(128 ** -0.5), C.c_float(0),
                             *map(C.c_int32, (0, 2, 2, 0, 2)), p(ws), C.c_size_t(need), C.c_int64(torch.cuda.current_stream().cuda_stream))
    assert L.b200_last_error() == 0
    ref = _reference(q, kc, vc, tables, lens, heads // kv_heads)
    assert float((out.double() - ref).norm() / ref.norm()) < 2.5e-3                # as in test_merge
