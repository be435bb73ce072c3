"""GPU parity of the tcgen05 form of latent decode at the edges of its tiles (128 tokens, two pages), chunks, head groups (16, 32, 64 columns, partly filled) and of the sink, against
float64.  Tolerance as in test_mla_chunks_gpu.py: probabilities and output are rounded to 16 bits, relative Frobenius below 2^-8 (bf16), 2^-11 (f16)."""
import numpy as np
import pytest
import torch

from candle_vllm_b200 import mla, seq_ops
from tests.gpu_util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,lens,loud", [
    (9, [127, 128, 129, 1, 64, 65], 1.0),                     # a group of 16 with seven heads too many; tiles of one page and of two
    (16, [191, 192, 193, 255, 256, 257, 384, 0], 1.0),        # chunks of 256 end inside a tile; a context of nothing
    (33, [700, 130], 4.0),                                    # 64 columns for 33 heads; loud scores: maxima move
    (100, [1300, 40, 600], 1.0),                              # two groups of 64, the second one with 36 heads
    (32, [9000, 100, 333], 1.0),                              # chunks of several tiles, the last one of one token
    (16, [300 + 7 * i for i in range(128)], 1.0),             # as many sequences as a warp adds up
])
def test_tiles_chunks_and_head_groups(dtype, heads, lens, loud):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(heads + len(lens))
    used = [-(-n // 64) for n in lens]
    pool = sum(used) + 1
    perm = np.random.default_rng(2).permutation(pool)
    tables, at = np.zeros((len(lens), max(used) + 3), np.int32), 0
    for i, n in enumerate(used):
        tables[i, :n] = perm[at:at + n]
        at += n
    mk = lambda *s, std=1.0: (torch.randn(s, device=DEV, generator=gen) * std).to(dtype)
    ckv, kpe, q, qp = mk(pool, 64, 1, 512), mk(pool, 64, 1, 64), mk(len(lens), heads, 512, std=0.3 * loud), mk(len(lens), heads, 64, std=0.3 * loud)
    sink = torch.randn(heads, device=DEV, generator=gen)
    scale = 192 ** -0.5
    ckv[int(perm[-1])] = kpe[int(perm[-1])] = float("nan")
    for i, n in enumerate(lens):                              # what lies past a context must not matter
        if n % 64:
            ckv[tables[i, used[i] - 1], n % 64:] = float("nan")
            kpe[tables[i, used[i] - 1], n % 64:] = float("nan")
    bt, cl = torch.from_numpy(tables).to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV)
    plain, with_sink = [], []
    for i, n in enumerate(lens):
        ids = torch.from_numpy(tables[i, :used[i]]).to(DEV).long()
        c, r = ckv[ids].flatten(0, 1)[:n, 0].double(), kpe[ids].flatten(0, 1)[:n, 0].double()
        s = (q[i].double() @ c.T + qp[i].double() @ r.T) * scale
        plain.append(torch.softmax(s, 1) @ c)
        with_sink.append(torch.softmax(torch.cat([s, sink.double()[:, None]], 1), 1)[:, :n] @ c)
    limit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    outs = [(mla.mla_paged_decode(q, qp, ckv, kpe, bt, cl, scale), plain)]
    if dtype == torch.bfloat16:
        outs.append((seq_ops.latent_attention_decode(q, qp, ckv, kpe, bt, cl, sink, scale), with_sink))
    for out, ref in outs:
        ref = torch.stack(ref)
        assert torch.isfinite(out).all()
        err = float((out.double() - ref).norm() / ref.norm())
        assert err < limit, err
