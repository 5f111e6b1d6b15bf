"""CPU: the native host steps read a fixed number of doubles per image, so arrays of another last axis are refused
(as NumPy's unpacking refused them) and arrays of another dtype are converted, never read as they lie."""

import numpy as np
import pytest

from cryojax_b200 import _native as nat
from cryojax_b200 import rotations as rot
from cryojax_b200 import simulator as S

CFG = S.BasicImageConfig((32, 32), 1.0, 300.0)


class OwnPose(S.AbstractPose):
    def __init__(self, q):
        self.q = q
        self.offset_in_angstroms = np.zeros(2)

    def quaternion(self):
        return self.q


def _reassigned(q):
    pose = S.QuaternionPose()
    pose.wxyz = q
    return pose


@pytest.mark.parametrize("make", [OwnPose, _reassigned])
@pytest.mark.parametrize("shape", [(), (0,), (3,), (5,), (12,), (1, 3), (4, 3), (3, 5), (3, 8), (3, 0)])
@pytest.mark.parametrize("n", [None, 1, 3])
def test_quaternions_of_another_length_are_refused(make, shape, n):
    with pytest.raises(ValueError):
        S.pack_image_params(make(np.ones(shape)), CFG, None, n=n)


def test_other_dtypes_are_converted():
    rng = np.random.default_rng(0)
    q = rng.standard_normal((5, 4)).astype(np.float32)
    want = rot.quat_to_matrix(rot.quat_normalize(q))
    records = nat.pack_image_params(5, q, np.zeros(2, np.float32), [np.float32(2.0), 300, np.ones(5, np.int64)],
                                    normalise=True)
    assert np.allclose(records[:, 0:9].reshape(-1, 3, 3), want, rtol=0, atol=1e-14)
    assert np.all(records[:, nat.P_PIXEL_SIZE] == 2.0) and np.all(records[:, nat.P_SCALE] == 1.0)
    single = want.astype(np.float32)
    assert np.array_equal(nat.orientation_order(single, 8), nat.orientation_order(single.astype(np.float64), 8))
    g = rng.standard_normal((5, 3, 2)).astype(np.float32)
    assert np.array_equal(nat.quaternion_grad(q, g), nat.quaternion_grad(q.astype(np.float64), g.astype(np.float64)))


@pytest.mark.parametrize("shape", [(9,), (3, 3), (5, 9), (5, 2, 3), (5, 3, 2), (5, 3, 4)])
def test_rotations_of_another_shape_are_refused(shape):
    with pytest.raises(ValueError):
        nat.orientation_order(np.ones(shape), 8)


@pytest.mark.parametrize("q,g", [((5, 3), (5, 3, 2)), ((3,), (1, 3, 2)), ((), (1, 3, 2)), ((5, 4), (5, 2, 2)),
                                 ((5, 4), (5, 6)), ((4, 4), (5, 3, 2))])
def test_quaternion_gradients_of_another_shape_are_refused(q, g):
    with pytest.raises(ValueError):
        nat.quaternion_grad(np.ones(q), np.ones(g))
