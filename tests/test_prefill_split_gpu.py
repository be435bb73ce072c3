"""GPU parity of the prompt-attention kernel where the CTAs of a cluster share a tile's keys (few tiles, cached prefixes), at the edges of the parts: key tiles that do not divide by the
parts, parts that a row or a whole M tile does not see, windows, the largest number of parts.  Reference, tolerance and their reasons as in test_prefill_umma_gpu.py; the merge adds
f32 rounding only."""
import numpy as np
import pytest
import torch

import candle_vllm_b200 as pkg
from tests.gpu_util import DEV
from tests.test_prefill_umma_gpu import _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,kvh,qlens,cached,window,loud", [
    (8, 2, [5], [8100], None, 1.0),                    # eight parts of eight key tiles
    (8, 2, [1, 1], [639, 767], None, 1.0),             # five and six key tiles: one part and three
    (32, 8, [100], [1950], None, 1.0),                 # 17 key tiles, the second M tile one token short of a third of its rows
    (4, 4, [250], [900], None, 6.0),                   # one head per tile: the first M tile's last row sees two key tiles less than the second one's; loud scores
    (4, 4, [256], [0], None, 1.0),                     # no prefix, two key tiles: not shared
    (8, 2, [64, 3, 40], [2000, 60, 700], None, 1.0),   # tiles of many keys and of few in one launch
    (8, 2, [60], [4000], 700, 1.0),                    # a window: its first key inside a page, six key tiles
    (8, 2, [64], [4000], 130, 1.0),                    # two or three key tiles, not shared in a launch of clusters
])
def test_parts_of_a_tile(dtype, H, kvh, qlens, cached, window, loud):
    g = torch.Generator(device=DEV)
    g.manual_seed(H * 100 + sum(qlens))
    klens = [a + b for a, b in zip(qlens, cached)]
    used = [-(-k // 64) for k in klens]
    pool = sum(used) + 1
    perm = np.random.default_rng(sum(klens)).permutation(pool)
    tables, at = [], 0
    for n in used:
        tables.append([int(x) for x in perm[at:at + n]])
        at += n
    mk = lambda *shape: torch.randn(shape, generator=g, device=DEV).to(dtype)
    q, k, v = mk(sum(qlens), H, 128) * loud, mk(sum(qlens), kvh, 128), mk(sum(qlens), kvh, 128)
    kc, vc = (torch.full((pool, 64, kvh, 128), float("nan"), dtype=dtype, device=DEV) for _ in range(2))
    for i, c in enumerate(cached):                     # everything of the pool that no context holds is NaN
        for j in range(-(-c // 64)):
            w = min(64, c - j * 64)
            kc[tables[i][j], :w], vc[tables[i][j], :w] = mk(w, kvh, 128), mk(w, kvh, 128)
    prep = pkg.prepare_prompt([list(range(n)) for n in klens], tables, 64, cached, chunk_size=max(qlens))
    _, _, meta = pkg.inputs.to_device(prep)
    op = pkg.PagedAttention(H, 128, 128 ** -0.5, kvh, sliding_window=window)
    out = op.forward(q, k, v, None, kc, vc, meta)
    again = op.forward(q, k, v, None, kc, vc, meta)
    ref = _reference(q, kc, vc, tables, qlens, klens, 128 ** -0.5, window)
    assert torch.isfinite(out).all() and torch.equal(out, again)
    err = float((out.double() - ref).norm() / ref.norm())
    assert err < (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11), err
