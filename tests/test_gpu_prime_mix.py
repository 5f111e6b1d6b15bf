"""GPU: sides with a prime factor above 7 beside sides without one.  Every kernel of the shared-memory FFT has an
instance with and one without prime stages, chosen by the lengths that it transforms: each pair of a volume side and
image sides here takes other instances in the column, row and post-processing passes.  Against the float64 oracle with
the tolerance of the slice and Ewald tests.
"""

import numpy as np
import pytest

from oracle import cryojax_oracle as O
from tests.helpers import IMAGE_REL_L2_TOL, make_volume, random_specs, rel_l2_per_image, specs_to_model_args

pytestmark = pytest.mark.gpu

# (box, image shape): the volume's side is 2 box
SIDES = [(22, (36, 40)), (24, (22, 35)), (24, (35, 22)), (22, (33, 26)), (24, (36, 40)), (32, (32, 26)), (32, (26, 32))]


@pytest.mark.parametrize("box,shape", SIDES)
@pytest.mark.parametrize("ewald", [False, True])
def test_images(cuda_device, box, shape, ewald):
    import torch

    from cryojax_b200 import simulator as S

    _, grid, fs = make_volume(box, 40, seed=box)
    specs = random_specs(3, seed=box + shape[0], shape=shape)
    pose, tt, cfg = specs_to_model_args(specs)
    vol = S.FourierVoxelGridVolume(torch.as_tensor(grid.astype(np.complex64)).cuda())
    integ = S.EwaldSphereExtraction(outputs_integral=False) if ewald else None
    model = S.make_image_model(vol, cfg, pose, tt, volume_integrator=integ)
    got = model.compute_fourier_image().cpu().numpy()
    ref = np.stack([O.compute_fourier_image(grid, fs, s, ewald=ewald) for s in specs])
    assert max(rel_l2_per_image(got, ref)) <= IMAGE_REL_L2_TOL
    got = model.simulate().cpu().numpy()
    ref = np.stack([O.simulate(grid, fs, s, ewald=ewald) for s in specs])
    assert max(rel_l2_per_image(got, ref)) <= IMAGE_REL_L2_TOL
