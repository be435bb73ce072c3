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
    assert rel_fro(y, ref) < 1e-3, rel_fro(y, ref)


@pytest.mark.parametrize("t", [pkg.GgmlType.Q4_K, pkg.GgmlType.Q6_K])
@pytest.mark.parametrize("rows", [512, 640, 2048])
@pytest.mark.parametrize("scales", ["small", "large", "mixed"])
def test_from_512_rows_a_weight_is_rounded_once(t, rows, scales):
    """unit rows of activations again: what comes back is the f32 weight rounded to f16, half a unit in the last place, whichever route takes the product"""
    n, k = 136, 2048
    rng = np.random.default_rng(rows)
    w = G.random_weight(rng, t, n, k).reshape(n * (k // 256), -1).copy()
    d = np.full(w.shape[0], {"small": 2e-4, "large": 0.02, "mixed": 2e-4}[scales], np.float16)
    if scales == "mixed":
        d[rng.random(w.shape[0]) < 0.03] = 0.02
    d = (d * rng.uniform(0.8, 1.2, d.shape)).astype(np.float16)          # scales whose products do not fit f16
    if t == pkg.GgmlType.Q4_K:
        w[:, 0:2] = d.view(np.uint8).reshape(-1, 2)
        w[:, 2:4] = (d * np.float16(0.37)).astype(np.float16).view(np.uint8).reshape(-1, 2)
    else:
        w[:, 208:210] = d.view(np.uint8).reshape(-1, 2)
    ref = G.dequantize_weight(w, t, n, k).astype(np.float64)
    mm = pkg.QMatMul.from_arc(pkg.QTensor.from_numpy(w.reshape(-1), t, (n, k)))
    # 2^-11 of the value or half of f16's smallest step; a 1/64 more for the second part of a Q6_K scale, which is rounded itself, far below
    bound = np.abs(ref) * 2.0 ** -11 * (1 + 1 / 64) + 2.0 ** -25 * (1 + 1 / 64) + (2.0 ** -25 if t == pkg.GgmlType.Q6_K else 0.0)
    for k0 in range(0, k, rows):
        count = min(rows, k - k0)
        x = torch.zeros(rows, k)
        x[torch.arange(count), k0 + torch.arange(count)] = 1.0
        y = mm.forward(x.to(DEV)).cpu().numpy().astype(np.float64)
        assert (np.abs(y[:count].T - ref[:, k0:k0 + count]) <= bound[:, k0:k0 + count]).all()


@pytest.mark.parametrize("t", [pkg.GgmlType.Q4_K, pkg.GgmlType.Q6_K])
@pytest.mark.parametrize("m,n", [(1024, 4096), (1025, 4096), (1152, 4096), (1153, 4096), (600, 9600), (700, 14336)])
def test_rounds_of_tiles_either_side_of_the_dense_path(t, m, n):
    """one rounding of the weights and one of the activations to f16, 2.0e-4 of a value each in the mean square, 2.9e-4 together, on either route; 3.45e-4 leaves no room for a
    second rounding of the weights"""
    k = 2048
    q = pkg.QTensor.from_numpy(G.random_weight(np.random.default_rng(m), t, n, k), t, (n, k))
    x = torch.randn(m, k, generator=torch.Generator(device=DEV).manual_seed(m), device=DEV)
    ref = x.double() @ pkg.dequantize(q).double().T
    err = float((pkg.QMatMul.from_arc(q).forward(x).double() - ref).norm() / ref.norm())
    assert err < 2.0 ** -11.5, err


@pytest.mark.parametrize("t", [pkg.GgmlType.Q4_K, pkg.GgmlType.Q6_K])
@pytest.mark.parametrize("m,n,k", [(65, 200, 2048), (200, 136, 4096), (256, 4096, 2048), (700, 384, 2048), (100, 20000, 2048)])
def test_accumulate_adds_to_what_is_there(t, m, n, k):
    """row tiles with the addend: clusters read, add and write; whole tiles of a CTA add in memory"""
    rng = np.random.default_rng(m)
    w = G.random_weight(rng, t, n, k)
    q = pkg.QTensor.from_numpy(w, t, (n, k))
    x = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float32)).to(DEV)
    start = torch.from_numpy(rng.standard_normal((m, n)).astype(np.float32)).to(DEV) * 3
    y, L = start.clone(), pkg.lib()
    ws = torch.empty(int(L.qmatmul_workspace_bytes(C.c_int32(m), C.c_int32(n), C.c_int32(k))), dtype=torch.uint8, device=DEV)
    L.qmatmul_f32(C.c_void_p(x.data_ptr()), C.c_void_p(q.data.data_ptr()), C.c_void_p(y.data_ptr()), C.c_int32(m), C.c_int32(n), C.c_int32(k), C.c_int32(t), C.c_int32(1),
                  C.c_void_p(ws.data_ptr()), C.c_size_t(ws.numel()), C.c_int64(torch.cuda.current_stream().cuda_stream))
    assert L.b200_last_error() == 0
    product = x.double() @ pkg.dequantize(q).double().T
    err = float(((y.double() - start.double()) - product).norm() / product.norm())
    assert err < 1e-3, err


@pytest.mark.parametrize("t,m", [(pkg.GgmlType.Q4_K, 100), (pkg.GgmlType.Q6_K, 200), (pkg.GgmlType.Q4_K, 600)])
def test_clusters_in_a_captured_graph(t, m):
    rng = np.random.default_rng(m)
    n, k = 640, 4096
    op = pkg.QMatMul.from_arc(pkg.QTensor.from_numpy(G.random_weight(rng, t, n, k), t, (n, k)))
    lin = pkg.Linear(torch.randn(1024, 640, device=DEV).bfloat16(), None)
    x = torch.randn(m, k, device=DEV)
    run = lambda: lin.forward(op.forward(x).bfloat16())
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        run()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = run()
    for seed in (1, 2):
        x.copy_(torch.randn(m, k, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, run())


def test_the_decode_kernel_leaves_registers_for_its_neighbours():
    """65536 registers an SM: 608 threads of 80 leave room for two blocks of 256 threads of 32 (rotation, norms, activation), of 96 for none"""
    assert 0 < pkg.lib().qmatmul_decode_kernel_registers(C.c_int32(pkg.GgmlType.Q4_K)) <= 80
