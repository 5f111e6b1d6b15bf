"""CPU: a pose's own offset array.  Its first two values are the shift and a third adds to the defocus where it is the
last; in an array of more than three values only the first two are read, and one of a single value is refused."""

import numpy as np
import pytest

from cryojax_b200 import _native as nat
from cryojax_b200 import simulator as S

CFG = S.BasicImageConfig((32, 32), 1.0, 300.0)
THEORY = S.ContrastTransferTheory(S.AstigmaticCTF(1.0e4))


def _pose(offset):
    pose = S.QuaternionPose()
    pose.offset_in_angstroms = offset
    return pose


@pytest.mark.parametrize("lead", [(), (3,)])
@pytest.mark.parametrize("width", [2, 3, 4, 7])
def test_widths(lead, width):
    offset = np.arange(1.0, 1.0 + np.prod(lead + (width,))).reshape(lead + (width,))
    p = S.pack_image_params(_pose(offset), CFG, THEORY)
    assert p.shape[0] == (lead or (1,))[0]
    assert np.array_equal(p[:, [nat.P_SHIFT_X, nat.P_SHIFT_Y]], offset[..., :2].reshape(-1, 2))
    height = offset[..., 2].reshape(-1) if width == 3 else 0.0
    assert np.array_equal(p[:, nat.P_DEFOCUS], np.broadcast_to(1.0e4 + height, p.shape[0]))


@pytest.mark.parametrize("shape", [(), (0,), (1,), (3, 1)])
def test_shorter_offsets_are_refused(shape):
    with pytest.raises((ValueError, IndexError)):
        S.pack_image_params(_pose(np.ones(shape)), CFG, THEORY)
