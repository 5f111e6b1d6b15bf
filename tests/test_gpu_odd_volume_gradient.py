"""GPU: the volume's gradient on the Ewald sphere at odd sides, which scatter straight into the gradient array (the
bricked accumulator takes x in pairs).  Every entry, summed against a random direction, and the largest entries one by
one, against float64 differences of the oracle; the loss is exactly quadratic in the volume, so central differences
have no truncation error.  Tolerances of test_gpu_ewald_grad (1e-4, single-precision sums of the scatter)."""

import numpy as np
import pytest

from oracle import cryojax_oracle as O
from tests.helpers import make_volume, random_specs
from tests.test_gpu_ewald_grad import GRAD_TOL, _loss, _model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,shape,layout", [(33, (32, 32), "bricked"), (41, (30, 26), "linear"), (33, (24, 40), "pairs"),
                                               (49, (48, 49), "pairs")])
def test_odd_side(cuda_device, side, shape, layout):
    from cryojax_b200.gradients import squared_residual_and_grad

    _, grid, fs = make_volume(side, 40, seed=side, pad_scale=1.0)
    assert grid.shape[0] == side
    specs = random_specs(2, seed=side + 1, shape=shape)
    rng = np.random.default_rng(side)
    obs = np.stack([O.simulate(grid, fs, s, ewald=True) for s in specs])
    obs = obs + rng.standard_normal(obs.shape) * obs.std()
    gg = squared_residual_and_grad(_model(grid, specs, layout=layout), obs, grid_grad=True)["d_grid"].cpu().numpy()

    def slope(direction):
        return (_loss(grid + direction, fs, specs, obs) - _loss(grid - direction, fs, specs, obs)) / 2

    size = np.abs(gg)
    for flat in np.argsort(size, axis=None)[::-1][:8]:
        at = np.unravel_index(flat, gg.shape)
        step = np.zeros_like(grid)
        step[at] = 1e-2 * max(abs(grid[at]), 1.0)
        want = (slope(step) + 1j * slope(1j * step)) / step[at].real
        assert abs(gg[at] - want) <= GRAD_TOL * abs(want), (at, gg[at], want)
    phase = np.exp(2j * np.pi * rng.uniform(size=grid.shape))
    direction = phase * np.abs(grid).max() * 1e-3
    want = slope(direction)
    got = float(np.sum((gg.conj() * direction).real))
    assert abs(got - want) <= GRAD_TOL * float(np.sqrt(np.sum(size**2 * np.abs(direction) ** 2)))
