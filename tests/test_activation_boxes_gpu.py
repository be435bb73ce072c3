"""The dequant-GEMM where activations come in boxes of a whole tile's rows: at the edges of the row tiles (one or two slices a stage, a last tile of few rows, more rows in the box than the
tensor has) and of the 64- and 32-row boxes of routed rows, against f64.  Tolerances and reasons as in test_moe_block_gpu.py: operands are rounded to f16, relative Frobenius 1e-3 a
product, 2e-3 for the block of three."""
import pytest
import torch

import candle_vllm_b200 as pkg
from tests.gpu_util import DEV
from tests.test_moe_block_gpu import _block, _weight

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [pkg.GgmlType.Q4_K, pkg.GgmlType.Q6_K])
@pytest.mark.parametrize("m", [33, 64, 65, 96, 97, 128, 129, 160, 225, 256, 257, 300, 513, 1000, 1408, 2048, 2049])
def test_row_tiles(t, m):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(m)
    n, k = 384, 2048
    data, w = _weight(gen, t, n, k)
    x = torch.randn((m, k), device=DEV, generator=gen)
    y = pkg.QMatMul.from_arc(pkg.QTensor(data, t, (n, k))).forward(x)
    ref = x.double() @ w.view(n, k).T
    err = float((y.double() - ref).norm() / ref.norm())
    assert torch.isfinite(y).all() and err < 1e-3, err


@pytest.mark.parametrize("T", [30, 40, 44, 64, 70, 100, 128, 129, 161])
def test_routed_rows(T):
    """every expert has every token: one chunk of 64 rows (up to 44 tokens), or chunks of up to 128"""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(T)
    E, H, I = 3, 512, 256
    (g, gd), (u, ud), (d, dd) = (_weight(gen, pkg.GgmlType.Q4_K, E * a, b) for a, b in ((I, H), (I, H), (H, I)))
    x, router = torch.randn((T, H), device=DEV, generator=gen), torch.randn((E, H), device=DEV, generator=gen) * 0.1
    types = (pkg.GgmlType.Q4_K,) * 3
    out = pkg.FusedMoe(router, g, u, d, types, E, H, I, E).forward(x)
    ref = _block(x.double(), router.double(), gd.view(E, I, H), ud.view(E, I, H), dd.view(E, H, I), E, E, True, None)
    err = float((out.double() - ref).norm() / ref.norm())
    assert err < 2e-3, err
