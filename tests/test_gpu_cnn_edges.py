"""GPU: the wide BF16 transpose and the four-channel col2im at sizes off their tiles, and where the general kernels
take over, against torch.  Both move or add the same values in the same order: transposes are exact, col2im is
compared in float32 before its one BF16 rounding (2^-9 relative)."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,ldi,ldo", [(1, 1, 8, 8), (64, 64, 64, 64), (63, 65, 72, 64), (200, 9, 16, 200),
                                               (129, 288, 288, 136), (37, 41, 41, 37), (72, 40, 41, 72)])
def test_transpose(cuda_device, rows, cols, ldi, ldo):
    import torch

    from cryojax_b200 import _native as nat

    x = torch.randn(rows, ldi, device="cuda").to(torch.bfloat16)
    out = torch.full((cols, ldo), 7.0, device="cuda", dtype=torch.bfloat16)
    nat.transpose_to_bf16(x, rows, cols, ldi, out, ldo)
    assert torch.equal(out[:, :rows], x[:, :cols].T)
    assert bool((out[:, rows:] == 7.0).all())


@pytest.mark.parametrize("h,w,c,extra", [(2, 2, 4, 0), (6, 4, 32, 0), (8, 10, 12, 4), (4, 4, 5, 3), (4, 6, 4, 1)])
@pytest.mark.parametrize("masked", [False, True])
def test_col2im(cuda_device, h, w, c, extra, masked):
    import torch

    from cryojax_b200 import _native as nat

    B, ldk = 3, 9 * c + extra
    dcol = torch.randn(B * (h // 2) * (w // 2), ldk, device="cuda")
    act = torch.randn(B, h, w, c, device="cuda").to(torch.bfloat16) if masked else None
    dx = torch.empty(B, h, w, c, device="cuda", dtype=torch.bfloat16)
    nat.cnn_col2im(dcol, ldk, act, B, h, w, c, dx)
    cols = dcol[:, :9 * c].reshape(B, (h // 2) * (w // 2), 9, c).permute(0, 3, 2, 1).reshape(B, c * 9, -1)
    want = torch.nn.functional.fold(cols, (h, w), 3, padding=1, stride=2).permute(0, 2, 3, 1)
    if masked:
        want = want * (act.float() > 0)
    assert torch.allclose(dx.float(), want, rtol=2**-8, atol=1e-6)
