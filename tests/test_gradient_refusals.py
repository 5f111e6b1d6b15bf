"""CPU: what the loss gradient refuses about the model, it refuses before it touches the observed images or a device."""

import numpy as np
import pytest

from cryojax_b200 import simulator as S
from cryojax_b200.gradients import squared_residual_and_grad


class Grid:
    shape = (64, 64, 64)
    device = "cpu"

    def get_representation(self):
        return self


CFG = S.BasicImageConfig((32, 32), 2.0, 300.0)
THEORY = S.ContrastTransferTheory(S.AstigmaticCTF(1.0e4))


def _model(pose=None, theory=THEORY, integrator=None, **kw):
    return S.LinearImageModel(Grid(), pose or S.QuaternionPose(), CFG, integrator or S.FourierSliceExtraction(), theory,
                              **kw)


@pytest.mark.parametrize("model,error", [
    (_model(theory=None, integrator=S.EwaldSphereExtraction()), NotImplementedError),
    (_model(translate_mode="atom"), ValueError),
    (_model(S.QuaternionPose(np.zeros(2), np.zeros(2), wxyz=np.ones((3, 4)))), ValueError),
])
def test_model_errors_come_first(model, error):
    with pytest.raises(error):
        squared_residual_and_grad(model, np.zeros((1, 32, 32), np.float32))
