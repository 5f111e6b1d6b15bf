"""GPU: packed observed images on either side of the multipliers' cache (72 KB: 135 x 68 entries fit, 136 x 69 do
not).  Packing without the contrast transfer scales every entry by the image's scale, and packing with it gives FP16
rows that are the single-precision ones over their RMS, rounded once (2^-11; subnormal halves 2^-25)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("py,px", [(134, 135), (135, 135), (135, 136), (136, 136), (128, 143), (128, 144)])
def test_rows_on_both_sides(cuda_device, py, px):
    import torch

    from cryojax_b200 import _native as nat
    from cryojax_b200 import simulator as S

    n, pxh = 3, px // 2 + 1
    rng = np.random.default_rng(py * px)
    pose = S.QuaternionPose(rng.uniform(-9, 9, n), rng.uniform(-9, 9, n), wxyz=rng.standard_normal((n, 4)))
    theory = S.ContrastTransferTheory(S.AstigmaticCTF(rng.uniform(8e3, 2e4, n), 200.0, 25.0))
    params = torch.as_tensor(S.pack_image_params(pose, S.BasicImageConfig((py, px), 2.0, 300.0), theory)).cuda()
    obs = torch.randn(n, py, pxh, dtype=torch.complex64, device="cuda")
    y32 = torch.empty(n, py, pxh, dtype=torch.complex64, device="cuda")
    z32 = torch.empty(n, py, pxh, device="cuda")
    y16 = torch.empty(n, py, pxh, 2, dtype=torch.float16, device="cuda")
    z16 = torch.empty(n, py, pxh, dtype=torch.float16, device="cuda")
    oo, oo16, yinv, zinv = (torch.empty(n, device="cuda") for _ in range(4))
    flags = nat.CJX_APPLY_CTF | nat.CJX_APPLY_TRANSLATION
    nat.pack_observed32(obs, params, py, px, flags, y32, z32, oo)
    nat.pack_observed(obs, params, py, px, flags, y16, z16, oo16, yinv, zinv)
    assert torch.equal(oo, oo16)
    assert torch.allclose(y16.float(), torch.view_as_real(y32) / yinv[:, None, None, None], rtol=2.0**-10, atol=2.0**-24)
    assert torch.allclose(z16.float(), z32 / zinv[:, None, None], rtol=2.0**-10, atol=2.0**-24)
