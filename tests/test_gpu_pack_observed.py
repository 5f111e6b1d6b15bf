"""GPU: the packed observed images at shapes with and without the multipliers' cache, narrow and wide rows.

Without contrast transfer the multiplier is the scale, so the single-precision rows are w O times it (two
roundings, 2^-23); with it the FP16 rows are the single-precision ones over their RMS, rounded once (2^-11) after
single-precision steps, and subnormal halves round to 2^-25.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("py,px", [(2, 2), (3, 2), (33, 31), (64, 64), (132, 132), (134, 134), (140, 150), (8, 600), (300, 5)])
def test_rows(cuda_device, py, px):
    import torch

    from cryojax_b200 import _native as nat
    from cryojax_b200 import simulator as S

    n, pxh = 5, px // 2 + 1
    rng = np.random.default_rng(py + px)
    pose = S.QuaternionPose(rng.uniform(-9, 9, n), rng.uniform(-9, 9, n), wxyz=rng.standard_normal((n, 4)))
    theory = S.ContrastTransferTheory(S.AstigmaticCTF(rng.uniform(8e3, 2e4, n), 200.0, 25.0))
    params = torch.as_tensor(S.pack_image_params(pose, S.BasicImageConfig((py, px), 2.0, 300.0), theory)).cuda()
    obs = torch.randn(n, py, pxh, dtype=torch.complex64, device="cuda")
    w = torch.full((py, pxh), 2.0, device="cuda")
    w[:, 0] = 1.0
    if px % 2 == 0:
        w[:, -1] = 1.0
    w[0, 0] = 0.0

    y32 = torch.empty(n, py, pxh, dtype=torch.complex64, device="cuda")
    z32 = torch.empty(n, py, pxh, device="cuda")
    oo = torch.empty(n, device="cuda")
    nat.pack_observed32(obs, params, py, px, 0, y32, z32, oo)
    assert torch.allclose(y32, w * obs, rtol=1e-6, atol=0) and torch.allclose(z32, w.expand(n, -1, -1))
    assert torch.allclose(oo, (w * obs.abs() ** 2).sum((1, 2)), rtol=1e-5)

    flags = nat.CJX_APPLY_CTF | nat.CJX_APPLY_TRANSLATION
    nat.pack_observed32(obs, params, py, px, flags, y32, z32, oo)
    y16 = torch.empty(n, py, pxh, 2, dtype=torch.float16, device="cuda")
    z16 = torch.empty(n, py, pxh, dtype=torch.float16, device="cuda")
    oo16, yinv, zinv = (torch.empty(n, device="cuda") for _ in range(3))
    nat.pack_observed(obs, params, py, px, flags, y16, z16, oo16, yinv, zinv)
    assert torch.equal(oo, oo16)
    want = torch.view_as_real(y32) / yinv[:, None, None, None]
    assert torch.allclose(y16.float(), want, rtol=2.0**-10, atol=2.0**-24)
    assert torch.allclose(z16.float(), z32 / zinv[:, None, None], rtol=2.0**-10, atol=2.0**-24)
    rms = torch.view_as_real(y32).square().mean((1, 2, 3)).sqrt()
    assert torch.allclose(torch.where(rms > 0, rms, torch.ones_like(rms)), yinv, rtol=1e-5)
