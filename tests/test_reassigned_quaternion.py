"""CPU: a quaternion assigned to a pose after its construction may be any sequence, as its normalisation takes it."""

import numpy as np
import pytest

from cryojax_b200 import simulator as S


@pytest.mark.parametrize("wxyz,batch", [([1.0, 0.0, 0.0, 0.0], None), ([[1.0, 0.0, 0.0, 0.0], [0.0, 2.0, 0.0, 0.0]], 2),
                                        (((1, 0, 0, 1),), 1)])
def test_sequences(wxyz, batch):
    pose = S.QuaternionPose()
    pose.wxyz = wxyz
    model = S.LinearImageModel(None, pose, S.BasicImageConfig((32, 32), 1.0, 300.0), S.FourierSliceExtraction(), None)
    assert model.batch_size == batch
    assert np.array_equal(model.image_params()[:, 0:9], S.pack_image_params(S.QuaternionPose(wxyz=np.array(wxyz, float)),
                                                                            model.image_config, None)[:, 0:9])
