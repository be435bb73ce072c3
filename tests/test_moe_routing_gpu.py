"""GPU parity of the routing of few tokens: the router's instances for up to 16 and 32 tokens either side of their borders, hidden sizes that leave a part less than
a whole batch of loads, the largest number of routed pairs of the one-launch plan; and the top-k on equal, zero and NaN probabilities.  Block: oracle and tolerance as in
test_moe_block_gpu.py.  Top-k: ids are exact (ties go to the smallest id); a weight is within 40 rounding steps of f32 of its f64 value (the sum of E <= 300 terms in
groups of 32, an exponential of 2 steps at arguments scaled by 1 step of up to 16)."""
import pytest
import torch

import candle_vllm_b200 as pkg
from candle_vllm_b200 import moe
from tests.gpu_util import DEV
from tests.test_moe_block_gpu import _block, _weight

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,topk,H", [(15, 33, 3, 2304), (16, 40, 4, 4352), (17, 33, 8, 2304), (31, 130, 5, 512), (32, 64, 32, 256), (33, 64, 4, 2304), (1, 2, 1, 256)])
def test_block_of_few_tokens(T, E, topk, H):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(T + E)
    I = 256
    (g, gd), (u, ud), (d, dd) = _weight(gen, 12, E * I, H), _weight(gen, 12, E * I, H), _weight(gen, 12, E * H, I)
    x = torch.randn((T, H), device=DEV, generator=gen)
    router = torch.randn((E, H), device=DEV, generator=gen) * 0.1
    out = pkg.FusedMoe(router, g, u, d, (12, 12, 12), E, H, I, topk).forward(x)
    ref = _block(x.double(), router.double(), gd.view(E, I, H), ud.view(E, I, H), dd.view(E, H, I), E, topk, True, None)
    assert float((out.double() - ref).norm() / ref.norm()) < 2e-3


@pytest.mark.parametrize("E", [4, 32, 33, 128, 200, 300])
def test_topk_of_equal_and_missing_probabilities(E):
    k, T = min(E, 8), 6
    gen = torch.Generator().manual_seed(E)
    logits = torch.randint(-2, 3, (T, E), generator=gen).float()              # many ties
    logits[1] = 0.0
    logits[2, 1:] = float("-inf")                                             # one expert has all of it, the others 0
    logits[3] = torch.randn(E, generator=gen) * 4
    logits[4, E // 2] = float("nan")                                          # never chosen while others are left
    w, ids = moe.topk_softmax(logits.to(DEV), k)
    w, ids = w.cpu(), ids.cpu().long()
    p = torch.softmax(logits.double(), 1)
    for t in range(T):
        v = logits[t].double().nan_to_num(float("-inf"), neginf=-1e30)
        want = sorted(range(E), key=lambda e: (-float(v[e]), e))[:k]
        if t == 4 and k == E:
            want = want[:-1]
        assert ids[t, :len(want)].tolist() == want
        if t == 4:
            assert torch.isnan(w[t]).all()
        else:
            assert ((w[t].double() - p[t, ids[t]]).abs() <= 40 * 2.0 ** -24 * p[t, ids[t]] + 1e-37).all()
