"""Dense GEMM above 64 rows: tiles that several CTAs share over k, with shares of the columns and of the k blocks that are not all alike, ragged
rows, columns and last k block, with and without a bias.  Oracle: fp64 matmul of the same 16-bit inputs.  Bound of an element: half a step of the
result (8 significant bits in bf16, 11 in f16: at most 2^-8 or 2^-11 of it; 2^-25 where f16 is subnormal) of the value that fp32 holds, which k additions
leave within k 2^-24 of the sum of the products' sizes."""
import pytest
import torch

import candle_vllm_b200 as pkg
from tests.gpu_util import DEV

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("m,n,k", [
    (65, 136, 2048),               # tiles of 64 columns, eight CTAs each
    (65, 1032, 1992),              # seven
    (65, 1496, 1992),              # five
    (129, 1032, 1992),             # three
    (129, 2048, 4104),             # two
    (129, 1496, 4104),             # tiles of 128 columns, five CTAs each
    (300, 1032, 4104),             # four
    (600, 1000, 4104),             # three
    (129, 6144, 512),              # tiles of one CTA
    (400, 6144, 512),              # pairs of SMs
])
def test_shared_tiles_match_oracle(dtype, bias, m, n, k):
    gen = torch.Generator().manual_seed(m * 31 + n + k)
    x = torch.randn((m, k), generator=gen).to(dtype).to(DEV)
    w = (torch.randn((n, k), generator=gen) / k ** 0.5).to(dtype).to(DEV)
    b = torch.randn(n, generator=gen).to(dtype).to(DEV) if bias else None
    linear = pkg.Linear(w, b)
    y = linear.forward(x)
    assert y.dtype == dtype and y.shape == (m, n)
    ref, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    if bias:
        ref, size = ref + b.double(), size + b.double().abs()
    half, summed = 2.0 ** (-8 if dtype == torch.bfloat16 else -11), size * (k * 2.0 ** -24)
    bound = (ref.abs() + summed) * half + 2.0 ** -25 + summed
    assert ((y.double() - ref).abs() <= bound).all()
    assert torch.equal(y, linear.forward(x))
