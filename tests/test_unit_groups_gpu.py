"""The dequant-GEMM's groups of warps take a CTA's units in turn, and its last tile is stored by all of them: ranges of fewer units than groups, tiles of one to four units (a tile
ends inside a round of the groups), tiles split between CTAs and whole ones, the last rows of a matrix, int4 scales that cannot be copied in 16-byte pieces."""
import numpy as np
import pytest
import torch

import candle_vllm_b200 as pkg
from oracle import ggml_quants as G
from oracle import gptq as OG
from tests.gpu_util import DEV, rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [pkg.GgmlType.Q4_K, pkg.GgmlType.Q6_K])
@pytest.mark.parametrize("m", [1, 32, 33, 64])
@pytest.mark.parametrize("n,k", [(130, 256), (20000, 256), (20100, 512), (20224, 768), (4224, 1024), (300, 2048), (80000, 2048)])
def test_ranges_and_tiles(t, m, n, k):
    if t == pkg.GgmlType.Q6_K and (k // 256 * 210) % 16:
        k = 2048
    rng = np.random.default_rng(n + m)
    q = pkg.QTensor.from_numpy(G.random_weight(rng, t, n, k), t, (n, k))
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).to(DEV)
    ref = x.double() @ pkg.dequantize(q).double().T
    y = pkg.QMatMul.from_arc(q).forward(x)
    # three roundings of a weight and one of an activation to f16, 2^-11 / sqrt(3) each in the mean square at most: 5.7e-4
    err = float((y.double() - ref).norm() / ref.norm())
    assert err < 8e-4, err


@pytest.mark.parametrize("m", [3, 40])
@pytest.mark.parametrize("n,k,g,size,shift", [(192, 256, 64, 0.01, 0), (192, 512, 128, 0.01, 0), (64, 768, -1, 0.01, 0), (320, 1024, 128, 0.01, 3), (320, 1024, 64, 0.2, 0), (128, 512, 64, 0.01, 1),
                                              (128, 512, -1, 0.2, 5)])
def test_int4_scales(m, n, k, g, size, shift):
    """shift: the scales start that many entries behind a 16-byte boundary; size 0.2: scales that the multiplication by 2^20 would take out of f16"""
    rng = np.random.default_rng(n + k + m)
    w = OG.pack_gptq(rng.integers(0, 16, (k, n), dtype=np.uint8))
    groups = 1 if g == -1 else k // g
    scales = torch.from_numpy(rng.uniform(0.3 * size, size, (groups, n)).astype(np.float32)).to(DEV).half()
    packed = pkg.marlin_permute_scales(scales, k, n, g)
    held = torch.empty(packed.numel() + 8, dtype=torch.float16, device=DEV)[shift:shift + packed.numel()].view_as(packed)
    held.copy_(packed)
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).to(DEV).half()
    y = pkg.gptq_matmul(x, pkg.marlin_weight_repack(torch.from_numpy(w.view(np.int32)).to(DEV), 4, False), held, None, None, torch.zeros(n, dtype=torch.int32, device=DEV), 4, g)
    ref = OG.gptq_matmul(x.float().cpu().numpy(), w, scales.float().cpu().numpy(), g)
    # f16 weights (offset and result rounded) and a result in f16: 2^-11 / sqrt(3) each in the mean square at most
    assert rel_fro(y.float().cpu().numpy(), ref) < 6e-4
