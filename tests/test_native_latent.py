"""Latent attention entered natively (csrc/py_calls.cpp) against the way through Python: the same results, the same refusals."""
import numpy as np
import pytest
import torch

import candle_vllm_b200 as pkg
from candle_vllm_b200 import _lib, mla
from tests.test_native_calls import through_python  # noqa: F401  (fixture)


def test_tensors_on_the_host_are_left_to_python():
    native = _lib.calls()
    if not native:
        pytest.skip("not built")
    c, r = torch.zeros(2, 512).half(), torch.zeros(2, 64).half()
    cc, rc = torch.zeros(3, 64, 1, 512).half(), torch.zeros(3, 64, 1, 64).half()
    assert native.latent_cache(c, r, cc, rc, torch.zeros(2, dtype=torch.int64)) is None
    assert native.latent_decode(torch.zeros(2, 16, 512).half(), torch.zeros(2, 16, 64).half(), cc, rc, torch.zeros(2, 3, dtype=torch.int32), torch.ones(2, dtype=torch.int32), 0.1) is None
    assert native.latent_cache(c) is None and native.latent_decode(1, 2, 3, 4, 5, 6, 7) is None


def _inputs(dtype, heads, lat=512):
    mk = lambda *s: (torch.randn(s, device="cuda") * 0.3).to(dtype)
    lens = [130, 1, 64, 300]
    tables = torch.from_numpy(np.random.default_rng(0).permutation(20).reshape(4, 5).astype(np.int32)).cuda()
    return dict(q=mk(4, heads, lat), qp=mk(4, heads, 64), cc=mk(20, 64, 1, lat), rc=mk(20, 64, 1, 64), bt=tables, lens=torch.tensor(lens, dtype=torch.int32, device="cuda"))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,lat", [(16, 512), (5, 512), (3, 128)])            # (both split-KV kernels and the generic one)
def test_results(through_python, dtype, heads, lat):  # noqa: F811
    d = _inputs(dtype, heads, lat)
    args = lambda **k: [{**d, **k}[n] for n in ("q", "qp", "cc", "rc", "bt", "lens")] + [0.07]
    strided = torch.randn(4, heads, 2 * lat, device="cuda").to(dtype)[..., ::2]
    for given in (args(), args(bt=d["bt"].long()), args(lens=d["lens"].long()), args(q=strided)):
        assert (_lib.calls().latent_decode(*given) is None) == (given is not None and (given[4].dtype != torch.int32 or given[5].dtype != torch.int32 or not given[0].is_contiguous()))
        assert torch.equal(mla.mla_paged_decode(*given), through_python(lambda: mla.mla_paged_decode(*given)))
    new, rot, slots = torch.randn(4, lat, device="cuda").to(dtype), torch.randn(4, 64, device="cuda").to(dtype), torch.tensor([3, -1, 700, 64], device="cuda")
    here, there = (d["cc"].clone(), d["rc"].clone()), (d["cc"].clone(), d["rc"].clone())
    assert _lib.calls().latent_cache(new, rot, *here, slots) == 0
    assert mla.concat_and_cache_mla(new, rot, *here, slots) is None
    through_python(lambda: mla.concat_and_cache_mla(new, rot, *there, slots))
    assert all(torch.equal(a, b) for a, b in zip(here, there)) and not torch.equal(here[0], d["cc"])


@pytest.mark.gpu
def test_refusals(through_python):  # noqa: F811
    d = _inputs(torch.bfloat16, 16)
    pos = torch.zeros(4, dtype=torch.int64, device="cuda")
    for call in (lambda: mla.mla_paged_decode(d["q"].half(), d["qp"], d["cc"], d["rc"], d["bt"], d["lens"], 0.1),
                 lambda: mla.concat_and_cache_mla(d["q"][:, 0].contiguous().half(), d["qp"][:, 0].contiguous(), d["cc"], d["rc"], pos),
                 lambda: mla.concat_and_cache_mla(torch.zeros(4, 12, device="cuda").bfloat16(), d["qp"][:, 0].contiguous(), torch.zeros(2, 64, 1, 12, device="cuda").bfloat16(), d["rc"], pos)):
        said = []
        for way in (lambda c: c(), through_python):
            with pytest.raises(pkg.BackendError) as e:
                way(call)
            said.append(str(e.value))
        assert said[0] == said[1]
