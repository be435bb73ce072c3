"""The natively entered operators (csrc/py_calls.cpp) against the way through Python: the same results, the same refusals, and None -- the Python way -- for arguments they are not made for.
The buffers that logits are read back to: lent while anything made from them is alive."""
import gc
import importlib.util
import os
import sys

import numpy as np
import pytest
import torch

import candle_vllm_b200 as pkg
from candle_vllm_b200 import _lib, llama
from oracle import ggml_quants as G


def test_host_rows_come_back_when_nothing_refers_to_them():
    rows = llama._HostRows(4, 6, pinned=False)
    a = rows.take(3)
    b = rows.take(4)
    c = rows.take(2)                                      # both are lent: an array of its own
    assert [x.shape for x in (a, b, c)] == [(3, 6), (4, 6), (2, 6)] and not rows.free
    a[:] = 1.0
    part = a[1]                                           # a view keeps the buffer, the array itself need not live
    del a, c
    gc.collect()
    assert not rows.free
    b[:] = 2.0
    assert (part == 1.0).all()
    del part
    gc.collect()
    assert len(rows.free) == 1
    del b
    gc.collect()
    assert len(rows.free) == 2
    many = llama._HostRows(1 << 12, 1 << 13, pinned=False)
    assert not many.free and many.take(2).shape == (2, 1 << 13)


def test_host_rows_are_pinned_when_they_are_needed(monkeypatch):
    made = []
    monkeypatch.setattr(llama.torch, "empty", lambda *a, pin_memory, **k: made.append(pin_memory) or torch.zeros(*a, **k))
    rows = llama._HostRows(4, 6)
    assert not made
    a = rows.take(2)
    assert made == [True]
    del a
    gc.collect()
    held = rows.take(3)
    assert made == [True] and held.shape == (3, 6)

    def refused(*a, **k):
        raise RuntimeError("out of memory")
    monkeypatch.setattr(llama.torch, "empty", refused)
    assert rows.take(4).shape == (4, 6)
    assert llama._HostRows(4, 6).take(1).shape == (1, 6)


def test_tensors_on_the_host_are_left_to_python():
    native = _lib.calls()
    if not native:
        pytest.skip("not built")
    x = torch.zeros(2, 8)
    assert native.silu_mul(x, x) is None
    assert native.linear(x.half(), torch.zeros(8, 8).half(), None) is None
    assert native.qmatmul(x, x, 8, 8, 12, None) is None
    assert native.silu_mul(1, x) is None and native.silu_mul(x) is None
    with pytest.raises(pkg.BackendError):
        pkg.Linear(torch.zeros(8, 8).half())


@pytest.fixture
def build_in(tmp_path):
    """build.py over a folder of its own that has a finished library and native calls of older sources"""
    spec = importlib.util.spec_from_file_location("b200_build_under_test", os.path.join(os.path.dirname(_lib.__file__), "build.py"))
    b = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(b)
    assert b.calls_path() == _lib._calls_path()
    b.HERE, b.CSRC, b.OBJ, b.SO = str(tmp_path), str(tmp_path), str(tmp_path / "obj"), str(tmp_path / "lib.so")
    for name in ("lib.so", b.calls_path(), "py_calls.cpp"):
        (tmp_path / name).write_text("")
    os.utime(b.calls_path(), (1, 1))
    return b


@pytest.mark.parametrize("missing", ["torch", "compiler", "headers"])
def test_the_library_is_built_without_native_calls(build_in, missing, monkeypatch, capfd):
    b = build_in
    stale = b.calls_path()
    if missing == "torch":
        monkeypatch.setitem(sys.modules, "torch", None)
    else:
        b.CCBIN = "/bin/false" if missing == "headers" else "/no/compiler"
    assert b.build() == b.SO
    assert os.path.exists(stale) == (missing == "torch") and "ctypes" in capfd.readouterr().err       # (whose it is cannot be known without torch)


def test_native_calls_of_another_torch_are_not_loaded(monkeypatch, tmp_path):
    native = _lib.calls()
    if not native:
        pytest.skip("not built")
    for name in ("_calls.so", os.path.basename(_lib._calls_path()), os.path.basename(_lib._SO)):
        (tmp_path / name).symlink_to(_lib._calls_path())
    monkeypatch.setattr(_lib, "_HERE", str(tmp_path))
    monkeypatch.setattr(_lib, "_SO", str(tmp_path / os.path.basename(_lib._SO)))
    for what, value in ((torch, "__version__"), (torch.version, "git_version"), (sys.implementation, "cache_tag")):
        with monkeypatch.context() as m:
            m.setattr(_lib, "_calls_module", None)
            m.setattr(what, value, "0123456789a")
            assert _lib.calls() is False


@pytest.fixture
def through_python(monkeypatch):
    """-> f(call): the call's result on the way through Python"""
    def run(call):
        with monkeypatch.context() as m:
            m.setattr(_lib, "_calls_module", False)
            return call()
    return run


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(3, 64), (64,), (2, 5, 64), (1, 1, 64)])
@pytest.mark.parametrize("bias", [False, True])
def test_linear(through_python, dtype, shape, bias):
    w = torch.randn(24, 64, device="cuda").to(dtype)
    op = pkg.Linear(w, torch.randn(24, device="cuda").to(dtype) if bias else None)
    for x in (torch.randn(*shape, device="cuda").to(dtype), torch.randn(*shape[:-1], 128, device="cuda").to(dtype)[..., ::2], torch.randn(*shape[:-1], 72, device="cuda").to(dtype)[..., 8:]):
        assert (_lib.calls().linear(x, op.weight, op.bias) is None) == (not x.is_contiguous())
        y = op.forward(x)
        assert y.shape == (*shape[:-1], 24) and torch.equal(y, through_python(lambda: op.forward(x)))
    for bad in (torch.randn(3, 64, device="cuda"), torch.randn(3, 56, device="cuda").to(dtype), torch.zeros(0, 64, device="cuda").to(dtype)):
        assert _lib.calls().linear(bad, op.weight, op.bias) is None


@pytest.mark.gpu
@pytest.mark.parametrize("t", [pkg.GgmlType.Q4_K, pkg.GgmlType.Q8_0])
@pytest.mark.parametrize("shape", [(512,), (3, 512), (2, 2, 512), (70, 512)])
def test_qmatmul_and_silu_mul(through_python, t, shape):
    q = pkg.QTensor.from_numpy(G.random_weight(np.random.default_rng(1), t, 130, 512), t, (130, 512))
    op = pkg.QMatMul.from_arc(q)
    x = torch.randn(*shape, device="cuda")
    assert _lib.calls().qmatmul(x, q.data, 130, 512, t, op._ws) is None          # no workspace yet
    y = [op.forward(x) for _ in range(2)]
    assert _lib.calls().qmatmul(x.half(), q.data, 130, 512, t, op._ws) is None
    ref = through_python(lambda: op.forward(x))
    assert y[0].shape == (*shape[:-1], 130) and all(float((a - ref).norm()) <= 1e-6 * float(ref.norm()) for a in y)      # (sums of split tiles in any order)
    u = torch.randn_like(ref)
    assert torch.equal(pkg.silu_mul(ref, u), through_python(lambda: pkg.silu_mul(ref, u)))
    assert torch.equal(pkg.silu_mul(ref.half(), u), through_python(lambda: pkg.silu_mul(ref.half(), u)))
    with pytest.raises(pkg.BackendError):
        op.forward(torch.randn(3, 256, device="cuda"))


@pytest.mark.gpu
@pytest.mark.parametrize("prompt", [False, True])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("strided", [False, True])
def test_paged_attention(through_python, prompt, fp8, strided):
    T, H, G_, hd, nb = 5, 8, 2, 128, 6
    gen = torch.Generator(device="cuda").manual_seed(3)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    q, kv = mk(T, H, hd), mk(T, 2, G_, hd)
    k, v = (kv[:, 0], kv[:, 1]) if strided else (kv[:, 0].contiguous(), kv[:, 1].contiguous())
    cache = [mk(nb, 64, G_, hd) for _ in range(2)]
    cache = [c.to(torch.float8_e4m3fn).view(torch.uint8) if fp8 else c for c in cache]
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    op = pkg.PagedAttention(H, hd, hd ** -0.5, G_, fp8_kvcache=fp8)
    if prompt:
        meta = pkg.InputMetadata(True, torch.arange(64, 64 + T, device="cuda"), i32([[1, 2]]), cu_seqlens_q=i32([0, T]), cu_seqlens_k=i32([0, T]), max_seqlen_q=T, max_seqlen_k=T)
    else:
        meta = pkg.InputMetadata(False, torch.arange(T, device="cuda") * 64 + 70, i32([[i, i + 1] for i in range(T)]), context_lens=i32([71] * T))

    def call(how):
        c = [x.clone() for x in cache]
        return [how(lambda: op.forward(q, k, v, None, c[0], c[1], meta)), *c]

    ref = call(through_python)
    for _ in range(2):
        assert all(torch.equal(a, b) for a, b in zip(call(lambda f: f()), ref))
    taken = _lib.calls().paged_attention(prompt, q, k, v, *cache, meta.slot_mapping, meta.block_tables, meta.context_lens, meta.cu_seqlens_q, meta.cu_seqlens_k, op._ws, H, G_, hd, T, 0, hd ** -0.5,
                                         0.0, fp8)
    assert torch.equal(taken, ref[0])                     # (K and V as parts of a fused projection as well)
    assert _lib.calls().paged_attention(prompt, q, k.transpose(0, 1), v.transpose(0, 1), *cache, meta.slot_mapping, meta.block_tables, meta.context_lens, meta.cu_seqlens_q, meta.cu_seqlens_k,
                                        op._ws, H, G_, hd, T, 0, hd ** -0.5, 0.0, fp8) is None
    if not prompt:
        with pytest.raises(pkg.BackendError):
            op.forward(q, k, v, None, cache[0], cache[1], pkg.InputMetadata(False, meta.slot_mapping, meta.block_tables, cu_seqlens_q=i32([0, T]), cu_seqlens_k=i32([0, T])))
    odd = pkg.PagedAttention(H, 72, 1.0, G_)              # a cache of another type than the model's: left to Python, which refuses it
    with pytest.raises(pkg.BackendError, match="cache dtype"):
        odd.forward(mk(T, H, 72), mk(T, G_, 72), mk(T, G_, 72), None, torch.zeros(nb, 64, G_, 72, dtype=torch.float32, device="cuda"), torch.zeros(nb, 64, G_, 72, dtype=torch.float32, device="cuda"), meta)


@pytest.mark.gpu
@pytest.mark.parametrize("prompt", [False, True])
def test_refusals_of_the_library(through_python, prompt):
    """what passes the native checks and is refused by the library comes back as its error, in the words of the way through Python"""
    T, H, G_, nb, native = 2, 4, 2, 4, _lib.calls()
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    mk = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device="cuda")

    def words(call):
        with pytest.raises(pkg.BackendError) as e:
            call()
        return str(e.value)

    hd = 264                                              # heads of more than 256
    op = pkg.PagedAttention(H, hd, 1.0, G_)
    meta = pkg.InputMetadata(prompt, torch.arange(T, device="cuda"), i32([[0]] * T), context_lens=i32([1, 2]), cu_seqlens_q=i32([0, T]), cu_seqlens_k=i32([0, T]), max_seqlen_q=T)
    call = lambda: op.forward(mk(T, H, hd), mk(T, G_, hd), mk(T, G_, hd), None, mk(nb, 64, G_, hd), mk(nb, 64, G_, hd), meta)
    ref = through_python(lambda: words(call))             # (makes the workspace)
    arguments = lambda: (prompt, mk(T, H, hd), mk(T, G_, hd), mk(T, G_, hd), mk(nb, 64, G_, hd), mk(nb, 64, G_, hd), meta.slot_mapping, meta.block_tables, meta.context_lens, meta.cu_seqlens_q,
                         meta.cu_seqlens_k, op._ws, H, G_, hd, T, 0, 1.0, 0.0, False)
    assert native.paged_attention(*arguments()) > 0 and words(call) == ref and ref.startswith("PagedAttention.forward: paged_attention")

    def pending():                                        # an error of an unchecked call of this thread is found by the check of the cache write
        pkg.lib().rms_norm(None, None, None, 1, 4, 0, 0, 0)
        return call()
    ref = through_python(lambda: words(pending))
    assert words(pending) == ref and ref.startswith("reshape_and_cache: rms_norm")
    pkg.lib().rms_norm(None, None, None, 1, 4, 0, 0, 0)
    assert native.paged_attention(*arguments()) < 0

    lin = pkg.Linear(mk(8, 64))
    x = mk(65)[1:]                                        # contiguous, on an odd multiple of two bytes
    assert native.linear(x, lin.weight, None) > 0 and words(lambda: lin.forward(x)) == through_python(lambda: words(lambda: lin.forward(x)))
    x, w, ws = torch.zeros(1, 256, device="cuda"), torch.zeros(144 * 8, dtype=torch.uint8, device="cuda"), torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    assert native.qmatmul(x, w, 8, 256, 99, ws) > 0 and b"type" in pkg.lib().b200_last_error_message()
    assert native.qmatmul(x, w, 8, 256, pkg.GgmlType.Q4_K, ws).shape == (1, 8)


@pytest.mark.gpu
def test_numbers_that_only_python_takes(through_python):
    """a window that is a float, a longest query that a decode step does not have: taken as they are on the way through Python, on the first call and, with the workspace there, on later ones"""
    T, H, G_, hd = 3, 8, 2, 128
    gen = torch.Generator(device="cuda").manual_seed(4)
    mk = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()
    q, k, v, kc, vc = mk(T, H, hd), mk(T, G_, hd), mk(T, G_, hd), mk(4, 64, G_, hd), mk(4, 64, G_, hd)
    i32 = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")
    meta = pkg.InputMetadata(False, torch.arange(T, device="cuda") + 70, i32([[0, 1]] * T), context_lens=i32([71, 72, 73]), max_seqlen_q=None)
    for window in (None, 4096.0, 20.0):
        op = pkg.PagedAttention(H, hd, hd ** -0.5, G_, sliding_window=window)
        ref = through_python(lambda: op.forward(q, k, v, None, kc, vc, meta))
        for _ in range(2):
            assert torch.equal(op.forward(q, k, v, None, kc, vc, meta), ref)
    native = _lib.calls()
    assert native.paged_attention(False, q, k, v, kc, vc, meta.slot_mapping, meta.block_tables, meta.context_lens, None, None, op._ws, H, G_, hd, None, 20.0, 1.0, 0.0, False) is None
    x, w = torch.zeros(1, 256, device="cuda"), torch.zeros(144 * 8, dtype=torch.uint8, device="cuda")
    assert native.qmatmul(x, w, 8.0, 256, 12, torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")) is None
