"""CPU: the native host steps (cjx_pack_image_params, cjx_orientation_order, cjx_quaternion_grad) against NumPy and
float64 autograd.

Tolerance: the same float64 formulas in another order of operations, 1e-14 relative; the order itself is exact.
"""

import numpy as np
import pytest

from cryojax_b200 import _native as nat
from cryojax_b200 import constants as C
from cryojax_b200 import gradients as G
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


@pytest.mark.parametrize("n,bits", [(0, 8), (1, 8), (2, 1), (700, 8), (5000, 3), (300, 13)])
def test_orientation_order(n, bits):
    rng = np.random.default_rng(n)
    records = np.zeros((n, 32))
    records[:, 0:9] = rot.quat_to_matrix(rng.standard_normal((n, 4))).reshape(n, 9)
    R = records[:, 0:9].reshape(-1, 3, 3)
    if n > 2:
        R[1] = np.diag([1.0, -1.0, -1.0])
        R[2] = [[0.0, 0.0, 1.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0]]  # a normal in the plane z = 0
    v = R[:, :, 2].copy()
    v[(v[:, 2] < 0) | ((v[:, 2] == 0) & (v[:, 1] < 0))] *= -1.0
    k = np.sqrt(2.0 / (1.0 + np.clip(v[:, 2], 0.0, 1.0)))
    scale = (1 << bits) - 1
    g = [np.clip(np.round((k * v[:, i] / np.sqrt(2.0) + 1.0) * 0.5 * scale), 0, scale) for i in (0, 1)]
    want = np.argsort(_hilbert(g[0], g[1], bits), kind="stable").astype(np.int32)
    got = S.orientation_order(R, bits)
    assert got.dtype == np.int32 and np.array_equal(got, want)


@pytest.mark.parametrize("offset_z", [False, True])
@pytest.mark.parametrize("batched", ["none", "pose", "all", "strided", "length one"])
def test_parameter_records(batched, offset_z):
    rng = np.random.default_rng(3)
    n = 1 if batched in ("none", "length one") else 6
    draw = {"none": lambda lo, hi: rng.uniform(lo, hi), "length one": lambda lo, hi: rng.uniform(lo, hi, 1),
            "pose": lambda lo, hi: rng.uniform(lo, hi), "all": lambda lo, hi: rng.uniform(lo, hi, n),
            "strided": lambda lo, hi: rng.uniform(lo, hi, (n, 3))[::-1, 1]}[batched]
    q = rng.standard_normal(4) if batched == "none" else rng.standard_normal((n, 4))
    off = (rng.uniform(-5, 5), rng.uniform(-5, 5)) if batched == "none" else rng.uniform(-5, 5, (2, n))
    z = draw(-50, 50) if offset_z else None
    pose = S.QuaternionPose(off[0], off[1], wxyz=q, offset_z_in_angstroms=z)
    ctf = S.AstigmaticCTF(draw(5e3, 2e4), draw(0, 500), draw(0, 180), draw(0.5, 3))
    theory = S.ContrastTransferTheory(ctf, S.FourierGaussian(draw(0.5, 2), draw(10, 80)), draw(0.05, 0.2), draw(0, 90))
    cfg = S.BasicImageConfig((32, 32), draw(1, 3), draw(100, 300))
    scale = draw(1, 2)
    p = S.pack_image_params(pose, cfg, theory, scale=scale)
    want = np.zeros((n, 32))
    want[:, 0:9] = np.reshape(rot.quat_to_matrix(rot.quat_normalize(q)), (-1, 9))
    want[:, 9], want[:, 10] = off
    df = np.asarray(ctf.defocus_in_angstroms) + (0.0 if z is None else z)
    ac, ps = theory.amplitude_contrast_ratio, np.deg2rad(theory.phase_shift)
    for k, v in ((11, df), (12, ctf.astigmatism_in_angstroms), (13, np.deg2rad(ctf.astigmatism_angle)),
                 (14, ctf.spherical_aberration_in_mm * 1e7), (15, C.wavelength_from_kilovolts(cfg.voltage_in_kilovolts)),
                 (16, ps + np.arctan(ac / np.sqrt(1 - ac**2))), (17, cfg.pixel_size), (18, scale),
                 (19, theory.envelope.amplitude), (20, theory.envelope.b_factor), (21, ac), (22, ps)):
        want[:, k] = v
    assert p.shape == (n, 32) and np.allclose(p, want, rtol=1e-14, atol=1e-15)
    bare = S.pack_image_params(pose, cfg, None, scale=scale, n=n)
    assert np.array_equal(bare[:, 0:9], p[:, 0:9]) and np.all(bare[:, 11:15] == 0) and np.all(bare[:, 19] == 1)


def test_inconsistent_batches_are_refused():
    cfg = S.BasicImageConfig((32, 32), 1.0, 300.0)
    with pytest.raises(ValueError):
        S.pack_image_params(S.QuaternionPose(np.zeros(3), np.zeros(3), wxyz=np.ones((3, 4))), cfg, None, scale=np.ones(2))
    with pytest.raises(ValueError):
        S.pack_image_params(S.QuaternionPose(0.0, 0.0, wxyz=np.ones((2, 2, 4))), cfg, None)
    with pytest.raises(nat.CryojaxB200Error):
        nat.orientation_order(np.zeros((1, 3, 3)), 0)


@pytest.mark.parametrize("columns", [2, 3])
def test_quaternion_gradient(columns):
    import torch

    rng = np.random.default_rng(columns)
    q, g = 3.0 * rng.standard_normal((50, 4)), rng.standard_normal((50, 3, columns))
    t = torch.tensor(q, requires_grad=True)
    (G._quat_to_matrix_t(t)[:, :, :columns] * torch.as_tensor(g)).sum().backward()
    assert np.allclose(nat.quaternion_grad(q, g), t.grad.numpy(), rtol=1e-13, atol=1e-14)
    assert np.allclose(nat.quaternion_grad(q[:1], g)[0], t.grad.numpy()[0], rtol=1e-13, atol=1e-14)
