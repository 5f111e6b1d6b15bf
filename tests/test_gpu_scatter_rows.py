"""GPU: the scatter with several steps per CTA and several CTAs per column of tiles, the last of them partial.

The number of steps grows with the batch (up to 8; one per CTA in the small batches that the large one is compared
with; with the volume's gradient 4 until the batch is four times as large).  N = 192 has 12 row tiles: 3 steps give 4
CTAs, 4 steps 3, 5 steps 3 with a partial last one and a sum flushed twice, 8 steps 2.  dL/dR sums 192 x 97 (slice) or 192 x 192 (Ewald) signed terms, at most four of a lane in single precision:
3 x 2^-24 of the terms' sizes, about sqrt(36864) = 192 times their sum: 3.5e-5, bound 5e-5 of the batch's largest.  The
volume's gradient is a single-precision sum in no fixed order: relative L2 2e-5.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOX = 96
ROW_TILES = 2 * BOX // 16


@pytest.mark.parametrize("steps", [3, 5, 8])
@pytest.mark.parametrize("surface,mode", [("slice", None), ("ewald", None), ("slice", 0), ("slice", 1), ("slice", 2),
                                          ("ewald", 1), ("ewald", 2)])
def test_large_batch_matches_small_batches(cuda_device, surface, mode, steps):
    import torch

    from cryojax_b200 import _native as nat
    from cryojax_b200 import simulator as S
    from cryojax_b200.gradients import squared_residual_and_grad

    column_tiles = ROW_TILES if surface == "ewald" else (BOX + 1 + 15) // 16
    tiles_per_slot = 32 if steps == 8 and mode is not None else steps
    n = -(-tiles_per_slot * 148 * 8 // (ROW_TILES * column_tiles))
    assert n * ROW_TILES * column_tiles // (148 * 8) == tiles_per_slot
    rng = np.random.default_rng(steps)
    torch.manual_seed(steps)
    vol = S.FourierVoxelGridVolume(torch.randn(2 * BOX, 2 * BOX, 2 * BOX, dtype=torch.complex64, device="cuda"))
    q, off, df = rng.standard_normal((n, 4)), rng.uniform(-5, 5, (n, 2)), rng.uniform(8e3, 2e4, n)
    observed = torch.randn(n, BOX, BOX, device="cuda")
    integrator = S.EwaldSphereExtraction(outputs_integral=False) if surface == "ewald" else None

    def gradients(i):
        pose = S.QuaternionPose(off[i, 0], off[i, 1], wxyz=q[i])
        model = S.make_image_model(vol, S.BasicImageConfig((BOX, BOX), 2.0, 300.0), pose,
                                   S.ContrastTransferTheory(S.AstigmaticCTF(df[i], 100.0, 30.0)),
                                   volume_integrator=integrator)
        return squared_residual_and_grad(model, observed[i], grid_grad=mode is not None)

    before = nat.tuning_get(nat.CJX_TUNE_SCATTER_VEC)
    try:
        if mode is not None:
            nat.tuning_set(nat.CJX_TUNE_SCATTER_VEC, mode)
        whole = gradients(slice(0, n))
        parts = [gradients(slice(s, s + 6)) for s in range(0, n, 6)]
    finally:
        nat.tuning_set(nat.CJX_TUNE_SCATTER_VEC, before)
    d_rot = np.concatenate([p["d_rotation"] for p in parts])
    assert np.abs(whole["d_rotation"] - d_rot).max() <= 5e-5 * np.abs(d_rot).max()
    if mode is not None:
        total = sum(p["d_grid"].to(torch.complex128) for p in parts)
        assert float((whole["d_grid"] - total).norm() / total.norm()) <= 2e-5
