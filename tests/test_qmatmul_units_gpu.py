"""Every weight of a GGML block, one by one: unit rows of activations give back the dequantised weights, so each quarter of a block, each offset of a Q6_K block
in its 16-byte groups (210 bytes a block: eight offsets over eight blocks) and both scale paths (block scales that fit f16 after the multiplication by a power of
two, and larger ones; the choice is made per warp of 32 rows) show in the output."""
import ctypes as C

import numpy as np
import pytest
import torch

import candle_vllm_b200 as pkg
from oracle import ggml_quants as G
from tests.gpu_util import DEV, rel_fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [pkg.GgmlType.Q4_K, pkg.GgmlType.Q6_K])
@pytest.mark.parametrize("rows", [32, 256])
@pytest.mark.parametrize("scales", ["small", "large", "mixed"])
def test_each_weight_comes_back(t, rows, scales):
    n, k = 136, 2048
    rng = np.random.default_rng(rows)
    w = G.random_weight(rng, t, n, k).reshape(n * (k // 256), -1).copy()
    d = np.full(w.shape[0], {"small": 2e-4, "large": 0.02, "mixed": 2e-4}[scales], np.float16)
    if scales == "mixed":
        d[rng.random(w.shape[0]) < 0.03] = 0.02                       # some warps hold such a row, most do not
    if t == pkg.GgmlType.Q4_K:
        w[:, 0:2] = d.view(np.uint8).reshape(-1, 2)
        w[:, 2:4] = d.view(np.uint8).reshape(-1, 2)
        term = d.astype(np.float64) * 63 * 15                         # largest product of a block that the sum holds
    else:
        w[:, 208:210] = d.view(np.uint8).reshape(-1, 2)
        term = np.abs(d.astype(np.float64)) * 128 * 32
    ref = G.dequantize_weight(w, t, n, k).astype(np.float64)
    mm = pkg.QMatMul.from_arc(pkg.QTensor.from_numpy(w.reshape(-1), t, (n, k)))
    # f16 rounding of the scale, of the offset and of the result, each at most half a unit in the last place of a value no larger than `term`
    bound = np.repeat(term.reshape(n, -1), 256, axis=1) * 3 * 2.0 ** -11 + 2.0 ** -24
    for k0 in range(0, k, rows):
        x = torch.zeros(rows, k)
        x[torch.arange(rows), k0 + torch.arange(rows)] = 1.0
        y = mm.forward(x.to(DEV)).cpu().numpy().astype(np.float64)
        assert (np.abs(y.T - ref[:, k0:k0 + rows]) <= bound[:, k0:k0 + rows]).all()


@pytest.mark.parametrize("t,m,k", [
    (pkg.GgmlType.Q4_K, 1025, 2048), (pkg.GgmlType.Q4_K, 2048, 2048), (pkg.GgmlType.Q4_K, 2049, 2048),      # the last rows of the dequant-GEMM, the first of the dense one
    (pkg.GgmlType.Q6_K, 1407, 2048), (pkg.GgmlType.Q6_K, 1408, 2048), (pkg.GgmlType.Q6_K, 512, 768),        # 768: no tensor-core form of the dequant-GEMM
    (pkg.GgmlType.Q8_0, 511, 512), (pkg.GgmlType.Q8_0, 512, 512),
])
def test_rows_on_either_side_of_the_dense_path(t, m, k):
    n = 200
    rng = np.random.default_rng(m)
    w = G.random_weight(rng, t, n, k)
    x = rng.standard_normal((m, k)).astype(np.float32)
    op = pkg.QMatMul.from_arc(pkg.QTensor.from_numpy(w, t, (n, k)))
    ref = G.qmatmul_dequant(x, w, t, n, k)
    y = op.forward(torch.from_numpy(x).to(DEV)).cpu().numpy()
    assert rel_fro(y, ref) < 1e-3, rel_fro(y, ref)             # both sides: weights and activations rounded to f16 once


def test_the_decode_kernel_leaves_registers_for_its_neighbours():
    """65536 registers an SM: 608 threads of 80 leave room for two blocks of 256 threads of 32 (rotation, norms, activation), of 96 for none"""
    assert 0 < pkg.lib().qmatmul_decode_kernel_registers(C.c_int32(pkg.GgmlType.Q4_K)) <= 80
