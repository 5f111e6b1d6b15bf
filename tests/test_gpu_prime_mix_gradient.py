"""GPU: the loss gradient on the Ewald sphere where only some of N, Py and Px have a prime factor above 7, so that the
adjoint's column, row and loss passes take different instances of the shared-memory FFT.

The slope of the loss along one random displacement of all the parameters (quaternion, offset, defocus, each by its own
typical step) against float64 central differences of the oracle.  Single precision holds each gradient to 1e-4 of its
group's size (test_gpu_ewald_grad), hence the slope to 1e-4 of the root of its summands' squares.
"""

import copy

import numpy as np
import pytest

from tests.test_gpu_ewald_grad import GRAD_TOL, _loss, _model, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box,shape", [(22, (36, 40)), (24, (22, 35)), (24, (35, 22)), (22, (33, 26)), (24, (36, 40)),
                                       (32, (32, 26)), (32, (26, 32))])
def test_slope_along_a_displacement(cuda_device, box, shape):
    from cryojax_b200.gradients import squared_residual_and_grad

    grid, og, fs, specs, obs = _setup(box, shape, 2, seed=7 * box + shape[0], kv=60.0)
    res = squared_residual_and_grad(_model(grid, specs), obs, grid_grad=False)
    rng = np.random.default_rng(box + shape[1])
    for b, s in enumerate(specs):
        q, t, f = 0.01 * rng.standard_normal(4), rng.standard_normal(2), 100.0 * rng.standard_normal()

        def loss_at(h):
            s2 = copy.deepcopy(s)
            s2.wxyz = s.wxyz + h * q
            s2.offset_in_angstroms = s.offset_in_angstroms + h * t
            s2.defocus_in_angstroms = s.defocus_in_angstroms + h * f
            return _loss(og, fs, [s2], obs[b:b + 1])

        want = (loss_at(2e-5) - loss_at(-2e-5)) / 4e-5
        parts = np.concatenate([res["d_wxyz"][b] * q, res["d_offset"][b] * t, [res["d_defocus"][b] * f]])
        assert abs(parts.sum() - want) <= GRAD_TOL * np.linalg.norm(parts), (b, parts, want)
