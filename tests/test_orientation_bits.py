"""CPU: the processing order at every number of bits per axis that NumPy's int64 arithmetic took, 1 to 32 (at 32 the
index's highest bit is the sign), NaN and infinite normals among the images; other numbers are refused."""

import numpy as np
import pytest

from cryojax_b200 import _native as nat
from cryojax_b200 import rotations as rot
from cryojax_b200 import simulator as S


def _hilbert(x, y, bits):
    x, y = x.astype(np.int64), y.astype(np.int64)
    d = np.zeros_like(x)
    s = 1 << (bits - 1)
    while s:
        rx, ry = (x & s) > 0, (y & s) > 0
        d += s * s * ((3 * rx) ^ ry)
        flip = ~ry & rx
        x, y = np.where(flip, s - 1 - x, x), np.where(flip, s - 1 - y, y)
        x, y = np.where(~ry, y, x), np.where(~ry, x, y)
        s >>= 1
    return d


@pytest.mark.parametrize("bits", [1, 7, 8, 16, 23, 24, 25, 28, 31, 32])
@pytest.mark.filterwarnings("ignore:invalid value")
def test_order_at_every_number_of_bits(bits):
    R = rot.quat_to_matrix(np.random.default_rng(bits).standard_normal((400, 4)))
    R[3, 0, 2] = R[7, 2, 2] = R[8, 1, 2] = np.nan
    R[9, 1, 2], R[11, 2, 2] = -np.inf, np.inf
    v = R[:, :, 2].copy()
    v[(v[:, 2] < 0) | ((v[:, 2] == 0) & (v[:, 1] < 0))] *= -1.0
    k = np.sqrt(2.0 / (1.0 + np.clip(v[:, 2], 0.0, 1.0)))
    scale = (1 << bits) - 1
    g = [np.clip(np.round((k * v[:, i] / np.sqrt(2.0) + 1.0) * 0.5 * scale), 0, scale) for i in (0, 1)]
    assert np.array_equal(S.orientation_order(R, bits), np.argsort(_hilbert(g[0], g[1], bits), kind="stable"))


@pytest.mark.parametrize("bits", [-1, 0, 33, 64])
def test_other_numbers_are_refused(bits):
    with pytest.raises(nat.CryojaxB200Error):
        S.orientation_order(np.eye(3), bits)


def test_a_fraction_is_refused():
    with pytest.raises(TypeError):
        S.orientation_order(np.eye(3), 8.5)
