"""GPU: the scatter's steps per CTA.  A large batch (several row tiles per CTA) gives each image the gradients that it
gets in a small one (one tile per CTA), with and without the volume's gradient.

dL/dR sums 64 x 33 signed single-precision terms, in double beyond at most four per lane: the two sums differ by at
most 3 x 2^-24 of the terms' sizes, about sqrt(2112) = 46 times the sum: 8e-6, bound 2e-5 of the batch's largest.
The volume's gradient is a single-precision sum in no fixed order, of about 1000 terms per voxel: the same bound on
its relative L2 difference.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("surface", ["slice", "ewald"])
@pytest.mark.parametrize("grid_grad", [False, True])
def test_large_batch_matches_small_batches(cuda_device, grid_grad, surface):
    import torch

    from cryojax_b200 import simulator as S
    from cryojax_b200.gradients import squared_residual_and_grad

    n, box = 832, 32
    rng = np.random.default_rng(5)
    torch.manual_seed(5)
    grid = torch.randn(2 * box, 2 * box, 2 * box, dtype=torch.complex64, device="cuda")
    vol = S.FourierVoxelGridVolume(grid)
    q, off = rng.standard_normal((n, 4)), rng.uniform(-5, 5, (n, 2))
    df = rng.uniform(8e3, 2e4, n)
    observed = torch.randn(n, box, box, device="cuda")
    integrator = S.EwaldSphereExtraction(outputs_integral=False) if surface == "ewald" else None

    def gradients(i):
        pose = S.QuaternionPose(off[i, 0], off[i, 1], wxyz=q[i])
        model = S.make_image_model(vol, S.BasicImageConfig((box, box), 2.0, 300.0), pose,
                                   S.ContrastTransferTheory(S.AstigmaticCTF(df[i], 100.0, 30.0)),
                                   volume_integrator=integrator)
        return squared_residual_and_grad(model, observed[i], grid_grad=grid_grad)

    whole = gradients(slice(0, n))
    parts = [gradients(slice(s, s + 16)) for s in range(0, n, 16)]
    d_rot = np.concatenate([p["d_rotation"] for p in parts])
    assert np.abs(whole["d_rotation"] - d_rot).max() <= 2e-5 * np.abs(d_rot).max()
    if grid_grad:
        total = sum(p["d_grid"].to(torch.complex128) for p in parts)
        assert float((whole["d_grid"] - total).norm() / total.norm()) <= 2e-5
