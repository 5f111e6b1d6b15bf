"""GPU: cjx_gemm's epilogue at the edges of its 32 x 32 blocks, for each output form and alignment, against float64.

Products of BF16 values are exact in FP32; a sum of K of them is off by at most K 2^-24 of the sum of their sizes
(accumulation order unknown: twice that), and a BF16 output by 2^-9 of its value more.  Columns beyond N keep theirs.
"""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,pad", [(1, 1, 8, 0), (33, 31, 72, 1), (129, 33, 8, 3), (130, 64, 200, 8), (1025, 288, 64, 0),
                                       (1030, 300, 1100, 4), (257, 96, 1088, 2)])
@pytest.mark.parametrize("form", ["float", "bf16", "bias relu bf16", "bias", "accumulate"])
def test_output_forms(cuda_device, m, n, k, pad, form):
    import torch

    from cryojax_b200 import _native as nat

    torch.manual_seed(m + n + k)
    ld = (k + 7) // 8 * 8  # the operands' row pitch
    a = torch.randn(m, ld, device="cuda").to(torch.bfloat16)
    b = torch.randn(n, ld, device="cuda").to(torch.bfloat16)
    bias = torch.randn(n, device="cuda") if "bias" in form else None
    dtype = torch.bfloat16 if "bf16" in form else torch.float32
    ldc = n + pad
    c = torch.full((m, ldc), 3.0, device="cuda", dtype=dtype)
    flags = (nat.CJX_GEMM_OUT_BF16 if "bf16" in form else 0) | (nat.CJX_GEMM_RELU if "relu" in form else 0)
    split = 1
    if form == "accumulate":
        flags, split = nat.CJX_GEMM_ACCUMULATE, 3
    nat.gemm(a, b, c, m=m, n=n, k=k, bias=bias, flags=flags, split_k=split)
    a, b = a[:, :k], b[:, :k]
    want = a.double() @ b.double().T
    size = a.double().abs() @ b.double().abs().T
    if bias is not None:
        want, size = want + bias.double(), size + bias.double().abs()
    if "relu" in form:
        want = want.clamp(min=0)
    if form == "accumulate":
        want, size = want + 3.0, size + 3.0
    bound = 2 * (k + 2) * 2.0 ** -24 * size + (2.0 ** -8 * want.abs() if "bf16" in form else 0.0)
    assert bool(((c[:, :n].double() - want).abs() <= bound).all())
    assert bool((c[:, n:] == 3.0).all())
