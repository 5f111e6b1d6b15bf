"""GPU: the shared-memory FFT's stages (cjx_fft_c2c) against numpy.fft in float64 at the lengths where they differ.

Lengths of one radix, of several, with one or two prime factors above 7
(a stage each, with few and with many outputs per lane), primes, and the ends
of the range.  Tolerance: a sequential single-precision sum of p/2 random
terms is off by about 0.3 eps sqrt(p) / 3 of its size (4e-7 at p = 1021), a
radix stage by about eps; 1e-6 relative L2 per row covers both.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 7, 9, 11, 12, 13, 22, 31, 45, 49, 77, 90, 121, 179, 180, 249, 331, 343, 358, 360, 720, 781, 961, 997,
         1001, 1018, 1021, 1022, 1023]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("direction", [-1, 1])
def test_every_kind_of_length(cuda_device, n, direction):
    import torch

    from cryojax_b200 import _native as nat

    rng = np.random.default_rng(1000 + n)
    x = (rng.standard_normal((19, n)) + 1j * rng.standard_normal((19, n))).astype(np.complex64)
    got = nat.fft_c2c(torch.as_tensor(x).cuda(), direction).cpu().numpy()
    xd = x.astype(np.complex128)
    ref = np.fft.fft(xd, axis=1) if direction < 0 else np.fft.ifft(xd, axis=1) * n
    err = np.linalg.norm(got - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert err.max() <= 1e-6, err.max()
