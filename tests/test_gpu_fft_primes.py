"""GPU: cjx_fft_c2c at lengths around the line between one and four outputs per lane of a prime stage (by the rounds
of 32 lanes that each takes), against numpy.fft in float64; tolerance as in test_gpu_fft_lengths."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [127, 131, 139, 158, 163, 202, 206, 254, 262, 302, 314, 338, 340, 352, 363, 476, 616, 676,
                               1003, 1007, 1009, 1013, 1016])
@pytest.mark.parametrize("direction", [-1, 1])
def test_lengths_around_the_line(cuda_device, n, direction):
    import torch

    from cryojax_b200 import _native as nat

    rng = np.random.default_rng(n)
    x = (rng.standard_normal((11, n)) + 1j * rng.standard_normal((11, n))).astype(np.complex64)
    got = nat.fft_c2c(torch.as_tensor(x).cuda(), direction).cpu().numpy()
    xd = x.astype(np.complex128)
    ref = np.fft.fft(xd, axis=1) if direction < 0 else np.fft.ifft(xd, axis=1) * n
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() <= 1e-6, err.max()
