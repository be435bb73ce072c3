"""GPU parity of the one-call expert block and of the row tiles of the grouped and plain dequant-GEMM at the sizes where they can go wrong, against float64 products of
the dequantised weights.  Tolerance: operands are rounded to f16 (2^-12 relative each, errors of the terms in quadrature): relative Frobenius 1e-3 per product, 2e-3
for the block of three."""
import pytest
import torch

import candle_vllm_b200 as pkg
from candle_vllm_b200 import moe, synthetic
from tests.gpu_util import DEV

pytestmark = pytest.mark.gpu


def _weight(gen, ggml_type, rows, k):
    w = synthetic.random_qtensor(gen, ggml_type, rows, k, DEV)
    return w.data, pkg.dequantize(w).double()


def _block(x, router, gate, up, down, E, topk, normalise, scaling):
    p = torch.softmax(x @ router.T, 1)
    w, ids = p.topk(topk, 1)
    w = (w / w.sum(1, keepdim=True) if normalise else w) * (scaling or 1.0)
    out = torch.zeros_like(x)
    for e in range(E):
        rows, slot = (ids == e).nonzero(as_tuple=True)
        if rows.numel():
            a = torch.nn.functional.silu(x[rows] @ gate[e].T) * (x[rows] @ up[e].T)
            out.index_add_(0, rows, w[rows, slot, None] * (a @ down[e].T))
    return out


@pytest.mark.parametrize("T,E,topk,H,I,types,normalise,scaling", [
    (1, 128, 8, 512, 256, (12, 12, 12), True, None),        # one token
    (16, 128, 8, 2048, 768, (12, 12, 12), True, None),      # decode: most experts have one row or none
    (32, 256, 8, 256, 256, (12, 12, 12), True, None),       # top-k in the plan's launch: one token per warp, every slot of a lane
    (5, 300, 4, 256, 256, (12, 12, 12), True, None),        # too many experts for it
    (7, 31, 3, 256, 256, (12, 12, 12), False, None),        # fewer experts than lanes
    (33, 5, 2, 256, 256, (12, 12, 12), False, 2.5),         # chunks of 32 with a remainder, experts not a multiple of the router's tile
    (63, 4, 2, 512, 512, (12, 12, 12), True, None),         # about 32 rows per expert, either side of a chunk
    (300, 4, 2, 256, 768, (12, 12, 12), True, 0.5),         # chunks of 128 with remainders
    (1100, 3, 3, 512, 256, (12, 12, 12), True, None),       # every expert has every token: several whole chunks
    (70, 8, 2, 2048, 2048, (14, 14, 14), True, None),       # the wider quantisation
    (40, 8, 2, 2048, 256, (12, 14, 12), True, None),        # gate and up of different types: two launches
    (20, 8, 1, 256, 256, (12, 12, 12), False, None),        # one expert per token
])
def test_block_matches_the_products(T, E, topk, H, I, types, normalise, scaling):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(T + E)
    (g, gd), (u, ud), (d, dd) = _weight(gen, types[0], E * I, H), _weight(gen, types[1], E * I, H), _weight(gen, types[2], E * H, I)
    x = torch.randn((T, H), device=DEV, generator=gen)
    router = torch.randn((E, H), device=DEV, generator=gen) * 0.1
    op = pkg.FusedMoe(router, g, u, d, types, E, H, I, topk, norm_topk_prob=normalise, routed_scaling_factor=scaling)
    assert op._block_covers(x, T)
    out = op.forward(x)
    ref = _block(x.double(), router.double(), gd.view(E, I, H), ud.view(E, I, H), dd.view(E, H, I), E, topk, normalise, scaling)
    err = float((out.double() - ref).norm() / ref.norm())
    assert err < 2e-3, err
    again = op.forward(x.t().contiguous().t())               # rows that are not contiguous are copied
    assert torch.equal(out, again)


def test_sort_is_stable_over_many_warps():
    gen = torch.Generator(device=DEV)
    gen.manual_seed(3)
    for P, E in [(1, 1), (31, 3), (1023, 128), (1025, 1024), (20000, 37), (40000, 1000)]:
        ids = torch.randint(0, E, (P,), device=DEV, generator=gen, dtype=torch.int32)
        e, s = moe.sort_expert_assignments(ids, E)
        want, order = torch.sort(ids.long(), stable=True)
        assert torch.equal(e.long(), want) and torch.equal(s.long(), order)


@pytest.mark.parametrize("ggml_type", [12, 14])
@pytest.mark.parametrize("m,n,k", [(65, 256, 2048), (96, 384, 2048), (127, 200, 2048), (128, 4096, 2048), (129, 128, 2048), (200, 1000, 4096), (257, 512, 2048), (511, 640, 2048)])
def test_row_tiles_of_the_dequant_gemm(ggml_type, m, n, k):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(m)
    data, w = _weight(gen, ggml_type, n, k)
    x = torch.randn((m, k), device=DEV, generator=gen)
    op = pkg.QMatMul(pkg.QTensor(data, ggml_type, (n, k)))
    ref = x.double() @ w.T
    for xin in (x, x.half()):                                # f32 activations (cast in the call) and the pre-cast entry
        err = float((op.forward(xin).double() - ref).norm() / ref.norm())
        assert err < 1e-3, err
