"""GPU: normalisation and mask at pixel counts on and off the 16-byte path, against float64.

A value is (x - mean) / std of single-precision x: rounding of x (2^-24 of its size, the images' largest value is a
few standard deviations) and two more single-precision steps, below 2e-6 of a standard deviation.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(2, 2), (5, 5), (6, 6), (7, 4), (31, 33), (64, 64), (200, 201)])
@pytest.mark.parametrize("masked", [False, True])
def test_normalised_images(cuda_device, shape, masked):
    import torch

    from cryojax_b200 import _native as nat

    rng = np.random.default_rng(shape[0])
    x = rng.standard_normal((3, *shape))
    f = np.fft.rfft2(np.fft.ifftshift(x, axes=(-2, -1)))
    mask = rng.uniform(0, 1, shape).astype(np.float32) if masked else None
    got = nat.postprocess_real(torch.as_tensor(f.astype(np.complex64)).cuda(), shape, shape, normalize=True, mask=mask)
    want = (x - x.mean(axis=(-2, -1), keepdims=True)) / x.std(axis=(-2, -1), keepdims=True)
    if masked:
        want = want * mask
    assert np.abs(got.cpu().numpy() - want).max() <= 1e-5  # the transform's own error, 1e-6 relative, on top
