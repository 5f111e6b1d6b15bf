"""GPU: the four-lane spline gather at one to four steps per CTA (the number grows with the batch) and at sides whose
last tile of columns or rows is nearly empty.  A sample's value does not depend on the CTA that takes it: an image of
a large batch has the bits that it has in a small one, which the float64 oracle checks to the forward tolerance."""

import numpy as np
import pytest

from oracle import cryojax_oracle as O
from tests.helpers import IMAGE_REL_L2_TOL, make_volume, random_specs, rel_l2_per_image, specs_to_model_args

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ewald", [False, True])
@pytest.mark.parametrize("box,batches", [(16, (300, 520, 800)), (17, (150, 300, 400)), (32, (90, 110, 140)),
                                         (40, (40, 60, 100))])
def test_batches_and_oracle(cuda_device, box, batches, ewald):
    import torch

    from cryojax_b200 import simulator as S

    shape = (box, box)
    _, grid, fs = make_volume(box, 30, seed=box)
    vol = S.FourierVoxelGridVolume(torch.as_tensor(grid.astype(np.complex64)).cuda())
    vol = S.FourierVoxelSplineVolume.from_fourier_voxel_grid(vol)
    specs = random_specs(max(batches), seed=box, shape=shape)

    def images(n):
        pose, tt, cfg = specs_to_model_args(specs[:n])
        integ = S.EwaldSphereExtraction(outputs_integral=False) if ewald else None
        return S.make_image_model(vol, cfg, pose, tt, volume_integrator=integ).compute_fourier_image()

    few = images(3)
    coefficients = O.compute_spline_coefficients(grid)
    ref = np.stack([O.compute_fourier_image(coefficients, fs, s, spline=True, ewald=ewald) for s in specs[:3]])
    assert max(rel_l2_per_image(few.cpu().numpy(), ref)) <= IMAGE_REL_L2_TOL
    for n in batches:
        many = images(n)
        assert torch.equal(many[:3], few)
        assert torch.equal(many[-3:], images(max(batches))[n - 3:n])
