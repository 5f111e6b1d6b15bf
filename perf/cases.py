"""Timed cases of the framework's public entry points: the calls that a particle-image program makes.

Seven kinds of call, each over the sizes that it meets in use:

  simulate  image models built from host parameters and simulated in one batched call, to Fourier or to real space
  batched   ``BatchedSimulator``: parameters uploaded and orientations sorted once, then images again and again
  gradient  ``squared_residual_and_grad`` against observed images, with or without the volume's gradient
  search    ``TemplateSharingSearch`` over an orientation grid, the best candidates rescored in single precision
  network   one gradient step of the pose-proposal network (forward and backward)

Volumes are sums of isotropic Gaussians, poses are uniform on SO(3), CTF parameters are uniform in the ranges of the
benchmark configurations.  ``exact`` restates every call in float64 with plain torch.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from cryojax_b200 import simulator as S

DEV = "cuda"
PIXEL = 2.0
KV = 300.0
AC = 0.1
CS_MM = 2.7


# ---- the cases -----------------------------------------------------------------------------------------------


def _sim(name, **kw):
    c = dict(name=name, kind="simulate", box=64, side=128, shape=64, padded=64, images=1, volume="grid",
             surface="slice", real=True, normalise=False, mask=False, envelope=False)
    c.update(kw)
    return c


def listed():
    return [
        # one particle looked at interactively, or the inner call of a program that handles images one at a time:
        # launches and host work are all there is
        _sim("one image 64"),
        # a small data set at once (the configuration of the plain benchmark: 128 images, pad factor 2)
        _sim("128 images 64 fourier", images=128, real=False),
        # a particle stack as it is written to disk: padded simulation, cropped, normalised and masked in real space
        _sim("stack 256 of 320 real", box=256, side=512, shape=256, padded=320, images=512, normalise=True, mask=True,
             envelope=True),
        # box sizes are what the microscope session gave, seldom a multiple of 32: 180^2 images from N = 360
        _sim("ragged 180", box=180, side=360, shape=180, padded=180, images=512, real=False),
        # the cubic-spline volume, for refinement programs that want a smooth interpolant
        _sim("spline 320", box=256, side=512, shape=320, padded=320, images=512, volume="spline", real=False),
        # the Ewald sphere at high resolution, large particles
        _sim("ewald 320", box=256, side=512, shape=320, padded=320, images=1024, surface="ewald", real=False),
        # the headline workload's images (320^2 from a 256^3 volume at pad factor 2), the parameters kept on the device
        dict(name="headline 320", kind="batched", boxes="256", shapes="320", images=2048, graph=False),
        # classes of different box sizes in one graph replay
        dict(name="mixed 96 to 256", kind="batched", boxes="96,128,192,256", shapes="96,128,192,256", images=512,
             graph=True),
        # volume reconstruction by gradient descent: pose, CTF and volume gradients
        dict(name="gradient volume 192", kind="gradient", box=192, images=1024, volume_gradient=True,
             surface="slice"),
        # local pose and defocus refinement: the same loss without the volume's gradient
        dict(name="gradient poses 256", kind="gradient", box=256, images=256, volume_gradient=False,
             surface="slice"),
        # global pose search of one batch of a data set: 768 directions x 48 in-plane angles
        dict(name="search 128", kind="search", box=128, images=1024, nside=8, inplane=48, top=8),
        # training of the proposal network
        dict(name="network step 128", kind="network", size=128, images=256, classes=768),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["simulate"] * 5 + ["batched"] * 2 + ["gradient"] * 2 + ["search", "network"])
    if kind == "simulate":
        box = _log_int(rng, 32, 256)  # any integer, odd ones and primes among them
        if rng.random() < 0.3:
            box = 32 * max(1, box // 32)
        pad = 1 if rng.random() < 0.15 else 2
        side = box * pad
        padded = box if pad == 1 or rng.random() < 0.5 else rng.randint(box, min(side, box + box // 3))
        shape = padded if rng.random() < 0.6 else rng.randint(max(16, (3 * padded) // 4), padded)
        volume = "spline" if rng.random() < 0.25 else "grid"
        surface = "ewald" if rng.random() < 0.25 else "slice"
        most = 2.0e7 if volume == "spline" else 6.0e7  # samples of the rotated plane
        most = min(most, 1.0e10 / side ** 2) if side < 100 else most
        images = _log_int(rng, 1, max(2, min(4096, most / (side * side))))
        real = rng.random() < 0.5
        return dict(kind=kind, box=box, side=side, shape=shape, padded=padded, images=images, volume=volume,
                    surface=surface, real=real, normalise=real and rng.random() < 0.5,
                    mask=real and rng.random() < 0.5, envelope=rng.random() < 0.3)
    if kind == "batched":
        n = rng.randint(1, 4)
        boxes = [_log_int(rng, 32, 192) if rng.random() < 0.5 else 32 * rng.randint(1, 6) for _ in range(n)]
        shapes = [b if rng.random() < 0.6 else rng.randint(b, b + b // 2) for b in boxes]
        most = 6.0e7 / sum(4 * b * b for b in boxes)
        return dict(kind=kind, boxes=",".join(map(str, boxes)), shapes=",".join(map(str, shapes)),
                    images=_log_int(rng, 4, max(5, min(1024, most))), graph=rng.random() < 0.5)
    if kind == "gradient":
        box = rng.choice([32, 64, 96, 128, 160, 192])
        surface = "ewald" if rng.random() < 0.25 else "slice"
        return dict(kind=kind, box=box, images=_log_int(rng, 2, max(4, min(1024, 6.0e7 / (4 * box * box)))),
                    volume_gradient=rng.random() < 0.6, surface=surface)
    if kind == "search":
        return dict(kind=kind, box=8 * rng.randint(4, 12), images=_log_int(rng, 16, 1024), nside=rng.choice([2, 4]),
                    inplane=rng.choice([12, 24, 36]), top=rng.choice([4, 8]))
    return dict(kind="network", size=rng.choice([64, 128]), images=8 * rng.randint(2, 31), classes=rng.choice([192, 768]))


def _gather_work(side, ncols, images, taps):
    """(bytes of distinct voxels, operations) of sampling `images` rotated planes."""
    samples = float(images) * side * ncols
    return 8.0 * min(float(side) ** 3, samples), samples * taps * 4.0


def _fft_ops(n):
    return 5.0 * n * math.log2(max(2, n))


def _image_work(side, py, images, volume, surface):
    half = side // 2 + 1
    ncols = side if surface == "ewald" else half
    b, f = _gather_work(side, ncols, images, 64 if volume == "spline" else 8)
    if py != side:
        rows = 1.0 if surface == "ewald" else 0.5
        f += images * (ncols * _fft_ops(side) + rows * py * (_fft_ops(side) + _fft_ops(py)) + (py // 2 + 1) * _fft_ops(py))
    return b, f + images * py * (py // 2 + 1) * 30.0


def work(case):
    k = case["kind"]
    if k == "simulate":
        b, f = _image_work(case["side"], case["padded"], case["images"], case["volume"], case["surface"])
        p = case["padded"]
        if case["real"]:
            out = 4.0 * case["shape"] ** 2
            f += case["images"] * 2.5 * p * p * math.log2(p * p)
        else:
            out = 8.0 * p * (p // 2 + 1)
        return {"bytes": b + case["images"] * (out + 256), "flops": f}
    if k == "batched":
        b = f = 0.0
        for box, p in zip(_ints(case["boxes"]), _ints(case["shapes"])):
            gb, gf = _image_work(2 * box, p, case["images"], "grid", "slice")
            b += gb + case["images"] * (8.0 * p * (p // 2 + 1) + 256)
            f += gf
        return {"bytes": b, "flops": f}
    if k == "gradient":
        p, n = case["box"], 2 * case["box"]
        b, f = _image_work(n, p, case["images"], "grid", case["surface"])
        b += case["images"] * (4.0 * p * p + 384)
        if case["volume_gradient"]:
            b += 16.0 * n ** 3
        return {"bytes": b, "flops": 2.5 * f}
    if k == "search":
        p = case["box"]
        t = 12 * case["nside"] ** 2 * case["inplane"]
        kp = p * (p // 2 + 1)
        return {"bytes": t * kp * 6.0 + case["images"] * 4.0 * p * p, "flops": 2.0 * case["images"] * t * kp * 3}
    layers, count = _layers(case["size"], case["classes"])
    per = sum(2.0 * L["k"] * L["cout"] * L["pixels"] for L in layers)
    return {"bytes": 8.0 * count + case["images"] * 2.0 * case["size"] ** 2, "flops": 3.0 * per * case["images"]}


# ---- inputs --------------------------------------------------------------------------------------------------


def _ints(text):
    return [int(v) for v in text.split(",")]


def _volume(box, rng):
    """Sum of isotropic Gaussians on a box^3 grid (float64, on the device)."""
    n = int(min(400, 20 + box))
    centre = rng.uniform(0.3 * box, 0.7 * box, (3, n))
    sigma = rng.uniform(1.0, 3.0, n) * min(1.0, box / 64.0) + 0.3
    amp = torch.as_tensor(rng.uniform(0.5, 1.5, n), device=DEV)
    x = torch.arange(box, device=DEV, dtype=torch.float64)
    g = [torch.exp(-((x[None] - torch.as_tensor(c, device=DEV)[:, None]) ** 2)
                   / (2.0 * torch.as_tensor(sigma, device=DEV)[:, None] ** 2)) for c in centre]
    out = torch.empty((box, box, box), dtype=torch.float64, device=DEV)
    for z0 in range(0, box, 64):
        a = (amp[:, None] * g[0][:, z0:z0 + 64])
        out[z0:z0 + 64] = (a.T @ (g[1][:, :, None] * g[2][:, None, :]).reshape(n, -1)).reshape(-1, box, box)
    return out


def _images_of(rng, n):
    q = rng.standard_normal((n, 4))
    return dict(q=q / np.linalg.norm(q, axis=1, keepdims=True), off=rng.uniform(-20.0, 20.0, (n, 2)),
                df=rng.uniform(5000.0, 25000.0, n), astig=rng.uniform(0.0, 500.0, n), angle=rng.uniform(0.0, 180.0, n),
                amp=rng.uniform(0.5, 1.5, n), b=rng.uniform(10.0, 80.0, n))


def _model(volume, p, shape, padded, *, surface="slice", envelope=False, normalise=False):
    pose = S.QuaternionPose(p["off"][:, 0], p["off"][:, 1], wxyz=p["q"])
    env = S.FourierGaussian(amplitude=p["amp"], b_factor=p["b"]) if envelope else None
    theory = S.ContrastTransferTheory(S.AstigmaticCTF(p["df"], p["astig"], p["angle"]), envelope=env)
    config = S.BasicImageConfig((shape, shape), PIXEL, KV, pad_options={"shape": (padded, padded)})
    integrator = S.EwaldSphereExtraction(outputs_integral=False) if surface == "ewald" else None
    return S.make_image_model(volume, config, pose, theory, volume_integrator=integrator, normalizes_signal=normalise)


def _soft_mask(shape):
    x = np.arange(shape) - shape // 2
    r = np.sqrt(x[:, None] ** 2 + x[None] ** 2)
    return (0.5 * (1.0 + np.cos(np.pi * np.clip((r - 0.4 * shape) / (0.08 * shape), 0.0, 1.0)))).astype(np.float32)


def _grid_volume(real, side):
    return S.FourierVoxelGridVolume.from_real_voxel_grid(real, pad_scale=side / real.shape[0])


def _sim_inputs(case, seed):
    rng = np.random.default_rng(seed)
    return _volume(case["box"], rng), _images_of(rng, case["images"])


def _batched_inputs(case, seed):
    rng = np.random.default_rng(seed)
    return [(_volume(b, rng), _images_of(rng, case["images"])) for b in _ints(case["boxes"])]


def _gradient_inputs(case, seed):
    """Volume, the parameters that the loss is taken at, and the observed images (SNR 0.1, real space, float32)."""
    rng = np.random.default_rng(seed)
    n, box = case["images"], case["box"]
    real = _volume(box, rng)
    p = _images_of(rng, n)
    near = dict(p)
    near["q"] = p["q"] + 0.02 * rng.standard_normal((n, 4))
    near["q"] /= np.linalg.norm(near["q"], axis=1, keepdims=True)
    near["off"] = p["off"] + rng.uniform(-2.0, 2.0, (n, 2))
    near["df"] = p["df"] + rng.uniform(-300.0, 300.0, n)
    clean = _real_space(_images64(_fourier64(real, 2 * box), p, box, surface=case["surface"]), box)
    return real, near, _noisy(clean, 0.1, seed)


def _search_inputs(case, seed):
    """Observed images at SNR 0.2 whose poses lie within about a degree of a grid orientation, so that the answer is
    not a coin toss between two grid points at the same distance."""
    rng = np.random.default_rng(seed)
    n, box = case["images"], case["box"]
    real = _volume(box, rng)
    table = _orientations(case)
    p = _images_of(rng, n)
    p["q"] = table[rng.integers(0, len(table), n)] + 0.004 * rng.standard_normal((n, 4))
    p["q"] /= np.linalg.norm(p["q"], axis=1, keepdims=True)
    p["off"] = rng.uniform(-4.0, 4.0, (n, 2))
    p["df"] = rng.uniform(8000.0, 20000.0, n)
    clean = _real_space(_images64(_fourier64(real, 2 * box), p, box), box)
    return real, p, _noisy(clean, 0.2, seed)


def _network_inputs(case, seed):
    rng = np.random.default_rng(seed)
    layers, count = _layers(case["size"], case["classes"])
    params = np.zeros(count, np.float32)
    for i, L in enumerate(layers):  # He initialisation, small biases
        std = math.sqrt((2.0 if i < len(layers) - 1 else 1.0) / L["k"])
        params[L["at"]:L["at"] + L["k"] * L["cout"]] = rng.standard_normal(L["k"] * L["cout"]) * std
        params[L["at"] + L["k"] * L["cout"]:L["at"] + (L["k"] + 1) * L["cout"]] = rng.standard_normal(L["cout"]) * 0.01
    x = torch.as_tensor(rng.standard_normal((case["images"], case["size"], case["size"])).astype(np.float32), device=DEV)
    labels = torch.as_tensor(rng.integers(0, case["classes"], case["images"]).astype(np.int32), device=DEV)
    near = torch.as_tensor(rng.integers(0, case["classes"], (case["classes"], 8)).astype(np.int32), device=DEV)
    return params, x.to(torch.bfloat16), labels, near


def _layers(size, classes):
    chans, out, at, s = (1, 32, 64, 128, 128, 256, 256), [], 0, size
    for cin, cout in zip(chans[:-1], chans[1:]):
        s //= 2
        out.append(dict(k=9 * cin, cin=cin, cout=cout, at=at, pixels=s * s))
        at += (9 * cin + 1) * cout
    for k, cout in ((256 * s * s, 512), (512, classes)):
        out.append(dict(k=k, cin=k, cout=cout, at=at, pixels=1))
        at += (k + 1) * cout
    return out, at


def _orientations(case):
    from cryojax_b200.healpix import OrientationGrid

    return OrientationGrid(case["nside"], case["inplane"]).quaternions()


def prepare(case, seed):
    k = case["kind"]
    if k == "simulate":
        real, p = _sim_inputs(case, seed)
        cls = S.FourierVoxelSplineVolume if case["volume"] == "spline" else S.FourierVoxelGridVolume
        volume = cls.from_real_voxel_grid(real, pad_scale=case["side"] / case["box"])
        volume.pair_grid()  # a program simulates from one volume many times: its device layout is made once
        return dict(case=case, volume=volume, p=p, mask=_soft_mask(case["shape"]) if case["mask"] else None)
    if k == "batched":
        from cryojax_b200.batched import BatchedSimulator

        models = [_model(_grid_volume(real, 2 * b), p, s, s) for (real, p), b, s in
                  zip(_batched_inputs(case, seed), _ints(case["boxes"]), _ints(case["shapes"]))]
        sim = BatchedSimulator(models, tuning=None)
        if case["graph"]:
            sim.capture()
        return dict(case=case, sim=sim)
    if k == "gradient":
        real, p, observed = _gradient_inputs(case, seed)
        box = case["box"]
        volume = _grid_volume(real, 2 * box)
        volume.bricked_grid() if case["volume_gradient"] else volume.pair_grid()
        return dict(case=case, volume=volume, p=p, observed=observed)
    if k == "search":
        from cryojax_b200 import rotations
        from cryojax_b200.search import TemplateSharingSearch

        real, p, observed = _search_inputs(case, seed)
        box = case["box"]
        model = _model(_grid_volume(real, 2 * box), p, box, box)
        search = TemplateSharingSearch(rotations.quat_to_matrix(_orientations(case)))
        search.build_templates(model)
        return dict(case=case, model=model, search=search, observed=observed)
    from cryojax_b200.pose_net import PoseProposalNet

    params, x, labels, near = _network_inputs(case, seed)
    net = PoseProposalNet(case["size"], case["classes"], max_batch=case["images"])
    net.load_state_dict({"params": params})
    return dict(case=case, net=net, x=x, labels=labels, near=near)


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "simulate":
        model = _model(state["volume"], state["p"], case["shape"], case["padded"], surface=case["surface"],
                       envelope=case["envelope"], normalise=case["normalise"])
        if case["real"]:
            return model.simulate(mask=state["mask"])
        return model.compute_fourier_image()
    if k == "batched":
        sim = state["sim"]
        return list(sim.replay() if case["graph"] else sim.run())
    if k == "gradient":
        from cryojax_b200.gradients import squared_residual_and_grad

        box = case["box"]
        model = _model(state["volume"], state["p"], box, box, surface=case["surface"])
        g = squared_residual_and_grad(model, state["observed"], grid_grad=case["volume_gradient"])
        # an optimiser keeps its parameters in single precision, in which the kernels compute
        out = {name: np.asarray(g[name], np.float32) for name in ("loss", "d_wxyz", "d_offset", "d_defocus")}
        if case["volume_gradient"]:
            out["d_grid"] = g["d_grid"]
        return out
    if k == "search":
        r = state["search"].run(state["model"], state["observed"], rerank_top=case["top"])
        return {"orientation": r.best_orientation, "score": r.best_score}
    net, b = state["net"], case["images"]
    logits = net.forward(state["x"], B=b)
    loss = net.backward(state["labels"], B=b, neighbours=state["near"], smoothing=0.2)
    return {"logits": logits, "loss": loss, "gradient": net.grads}


# ---- the same in float64 -------------------------------------------------------------------------------------


def _fourier64(real, side):
    """Centred full FFT of the volume zero-padded to side^3 (complex128)."""
    d = real.shape[0]
    extra = side - d
    left = extra // 2 + (1 if side % 2 == 0 and d % 2 == 1 else 0)
    padded = torch.zeros((side,) * 3, dtype=torch.complex128, device=DEV)
    padded[left:left + d, left:left + d, left:left + d] = real
    return torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(padded)))


def _spline64(grid):
    """Cubic-spline coefficients: per axis the end values / 6, tridiag(1, 4, 1) inside, linear extrapolation outside."""
    n = grid.shape[0]
    inner = torch.linalg.inv(4.0 * torch.eye(n - 2, dtype=torch.float64, device=DEV)
                             + torch.diag(torch.ones(n - 3, dtype=torch.float64, device=DEV), 1)
                             + torch.diag(torch.ones(n - 3, dtype=torch.float64, device=DEV), -1))
    m = torch.zeros((n + 2, n), dtype=torch.float64, device=DEV)
    m[1, 0] = m[n, n - 1] = 1.0 / 6.0
    m[2:n, 1:n - 1] = inner
    m[2:n, 0] -= inner[:, 0] / 6.0
    m[2:n, n - 1] -= inner[:, -1] / 6.0
    m[0] = 2.0 * m[1] - m[2]
    m[n + 1] = 2.0 * m[n] - m[n - 1]
    out = grid
    for _ in range(3):  # each pass transforms the last axis and moves it to the front
        re, im = out.real.reshape(-1, n) @ m.T, out.imag.reshape(-1, n) @ m.T
        out = torch.complex(re, im).reshape(*out.shape[:2], n + 2).permute(2, 0, 1).contiguous()
    return out


def _rotation64(q):
    q = q / torch.linalg.norm(q, dim=-1, keepdim=True)
    w, x, y, z = q.unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1).reshape(*q.shape[:-1], 3, 3)


def _wavelength():
    v = 1000.0 * KV
    return 12.2639 / math.sqrt(v + 0.97845e-6 * v * v)


def _taps(off, n, m, taps):
    """(index, inside, weight) per tap along one axis at offsets `off` from the centre; a negative index wraps once."""
    low = torch.floor(off).detach()
    f = off - low
    if taps == 2:
        ws = [1.0 - f, f]
    else:
        g = 1.0 - f
        ws = [g ** 3, 4 - 6 * f ** 2 + 3 * f ** 3, 4 - 6 * g ** 2 + 3 * g ** 3, f ** 3]
    out = []
    for t, w in enumerate(ws):
        i = low.to(torch.int64) + n // 2 + t
        i = torch.where(i < 0, i + m, i)
        ok = (i >= 0) & (i < m)
        out.append((torch.where(ok, i, 0), ok, w))
    return out


def _sample64(grid, rot, n, surface, corners=None):
    """Rotated planes [b, v, u] of a voxel grid (side n) or of spline coefficients (side n + 2)."""
    m = grid.shape[0]
    u = torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=torch.float64)
    v = u[:, None]
    u = u if surface == "ewald" else torch.arange(n // 2 + 1, device=DEV, dtype=torch.float64) * torch.where(
        torch.arange(n // 2 + 1, device=DEV) < n - n // 2, 1.0, -1.0)
    u = u[None]
    off = [rot[:, a, 0, None, None] * u + rot[:, a, 1, None, None] * v for a in range(3)]
    if surface == "ewald":
        w = _wavelength() / (2.0 * n * PIXEL) * (u * u + v * v)
        off = [o + rot[:, a, 2, None, None] * w for a, o in enumerate(off)]
    x, y, z = (_taps(o, n, m, 2 if m == n else 4) for o in off)
    flat, out = grid.reshape(-1), 0.0
    for iz, oz, wz in z:
        for iy, oy, wy in y:
            row, okr, wr = (iz * m + iy) * m, oz & oy, wz * wy
            for ix, ox, wx in x:
                idx, ok, w = row + ix, okr & ox, wr * wx
                out = out + w * torch.where(ok, flat[idx], 0.0)
                if corners is not None:
                    corners.append((idx, torch.where(ok, w, 0.0).detach()))
    return out


def _crop64(x, p, dims):
    n = x.shape[dims[0]]
    x = torch.fft.fftshift(x, dim=dims)
    for d in dims:
        x = x.narrow(d, n // 2 - p // 2, p)
    return torch.fft.ifftshift(x, dim=dims)


def _irfft2(f, shape):
    """Inverse of rfft2 that ignores what a real image cannot have in its first and Nyquist columns."""
    t = torch.fft.ifft(f, dim=-2)
    keep = torch.ones(f.shape[-1], dtype=torch.float64, device=DEV)
    keep[0] = 0.0
    if shape % 2 == 0:
        keep[-1] = 0.0
    return torch.fft.irfft(torch.complex(t.real, t.imag * keep), n=shape, dim=-1)


def _chi_cycles(p, sl, qx, qy):
    lam = _wavelength()
    df, astig, ang = (_col(p, k, sl) for k in ("df", "astig", "angle"))
    k2 = qx * qx + qy * qy
    theta = torch.atan2(qx.expand_as(k2), qy.expand_as(k2))
    d = df + 0.5 * astig * torch.cos(2.0 * (theta - ang * math.pi / 180.0))
    return -0.5 * d * lam * k2 + 0.25 * CS_MM * 1e7 * lam ** 3 * k2 * k2


def _col(p, k, sl):
    v = p[k][sl]
    v = v if isinstance(v, torch.Tensor) else torch.as_tensor(v, device=DEV)
    return v[:, None, None]


def _finish64(planes, n, p, sl, py, surface, envelope):
    """Resize, contrast transfer, envelope and translation: rfft images [b, py, py//2+1] of the sampled planes."""
    h = n // 2
    if surface == "slice":
        if py == n:
            f = planes.clone()
            if n % 2 == 0:
                for i, j in ((h, 0), (0, h), (h, h)):
                    f[:, i, j] = f[:, i, j].real.to(f.dtype)
        else:
            f = torch.fft.rfft2(_crop64(_irfft2(planes, n), py, (-2, -1)))
    else:
        o = planes if py == n else torch.fft.fft2(_crop64(torch.fft.ifft2(planes), py, (-2, -1)))
    qx = torch.fft.rfftfreq(py, PIXEL, device=DEV, dtype=torch.float64)[None, None]
    qy = torch.fft.fftfreq(py, PIXEL, device=DEV, dtype=torch.float64)[None, :, None]
    chi = 2.0 * math.pi * _chi_cycles(p, sl, qx, qy)
    if surface == "slice":
        f = f * torch.sin(chi - math.atan(AC / math.sqrt(1.0 - AC * AC)))
    else:
        w = py // 2 + 1
        pos = o[..., :w].clone()
        neg = torch.roll(torch.flip(o, (-2, -1)), (1, 1), (-2, -1))[..., :w].clone()
        if py % 2 == 0:
            pos[..., -1] = torch.conj(neg[..., -1])
            neg[:, py // 2, 0] = pos[:, py // 2, 0]
            pos[:, py // 2, 0] = torch.conj(pos[:, py // 2, 0])
        w1, w2 = AC, math.sqrt(1.0 - AC * AC)
        sr, si = pos.real + neg.real, pos.imag + neg.imag
        dr, di = neg.real - pos.real, pos.imag - neg.imag
        sn, cs = torch.sin(chi), torch.cos(chi)
        im = (w2 * di + w1 * dr) * sn + (w2 * dr - w1 * di) * cs
        if py % 2 == 0:
            flip = torch.ones((py, w), dtype=torch.float64, device=DEV)
            flip[py // 2, 0] = -1.0
            im = im * flip
        f = 0.5 * torch.complex((w2 * sr + w1 * si) * sn + (w2 * si - w1 * sr) * cs, im)
    if envelope:
        f = f * (_col(p, "amp", sl) * torch.exp(-0.25 * _col(p, "b", sl) * (qx * qx + qy * qy)))
    off = p["off"][sl]
    off = off if isinstance(off, torch.Tensor) else torch.as_tensor(off, device=DEV)
    ph = -2.0 * math.pi * (qx * off[:, 0, None, None] + qy * off[:, 1, None, None])
    keep = torch.ones((py, py // 2 + 1), dtype=torch.float64, device=DEV)
    if py % 2 == 0:
        keep[py // 2, 0] = keep[0, -1] = keep[py // 2, -1] = 0.0
    return f * torch.complex(torch.cos(ph), torch.sin(ph)) * keep


def _images64(grid, p, py, *, side=None, surface="slice", envelope=False):
    n = side or grid.shape[0]
    count = len(p["df"])
    step = max(1, int(2.5e7 // (n * n)))
    rot = _rotation64(torch.as_tensor(p["q"], device=DEV))
    out = torch.empty((count, py, py // 2 + 1), dtype=torch.complex128, device=DEV)
    for s in range(0, count, step):
        sl = slice(s, min(count, s + step))
        out[sl] = _finish64(_sample64(grid, rot[sl], n, surface), n, p, sl, py, surface, envelope)
    return out


def _real_space(f, py):
    return torch.fft.fftshift(_irfft2(f, py), dim=(-2, -1))


def _noisy(clean, snr, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 1)
    sd = torch.sqrt(clean.var(dim=(-2, -1), unbiased=False, keepdim=True) / snr)
    return (clean + sd * torch.randn(clean.shape, generator=g, device=DEV, dtype=torch.float64)).float()


def _exact_simulate(case, seed):
    real, p = _sim_inputs(case, seed)
    grid = _fourier64(real, case["side"])
    if case["volume"] == "spline":
        grid = _spline64(grid)
    py, sh = case["padded"], case["shape"]
    f = _images64(grid, p, py, side=case["side"], surface=case["surface"], envelope=case["envelope"])
    if not case["real"]:
        return f
    x = _real_space(f, py)
    lo = py // 2 - sh // 2
    x = x[:, lo:lo + sh, lo:lo + sh]
    if case["normalise"]:
        x = (x - x.mean(dim=(-2, -1), keepdim=True)) / x.std(dim=(-2, -1), unbiased=False, keepdim=True)
    if case["mask"]:
        x = x * torch.as_tensor(_soft_mask(sh), device=DEV).double()
    return x


def _exact_gradient(case, seed):
    real, p, observed = _gradient_inputs(case, seed)
    py, n, count = case["box"], 2 * case["box"], case["images"]
    grid = _fourier64(real, n)
    leaf = {k: torch.as_tensor(p[k], device=DEV).clone().requires_grad_(True) for k in ("q", "off", "df")}
    fixed = {k: torch.as_tensor(p[k], device=DEV) for k in ("astig", "angle")}
    d_grid = torch.zeros((n ** 3, 2), dtype=torch.float64, device=DEV)
    loss = torch.empty(count, dtype=torch.float64, device=DEV)
    step = max(1, int(1.0e7 // (n * n)))
    for s in range(0, count, step):
        sl = slice(s, min(count, s + step))
        corners = [] if case["volume_gradient"] else None
        planes = _sample64(grid, _rotation64(leaf["q"][sl]), n, case["surface"], corners)
        planes.retain_grad()
        q = {**fixed, "off": leaf["off"], "df": leaf["df"]}
        x = _real_space(_finish64(planes, n, q, sl, py, case["surface"], False), py)
        each = ((x - observed[sl].double()) ** 2).sum(dim=(-2, -1))
        each.sum().backward()
        loss[sl] = each.detach()
        if corners is not None:
            g = torch.view_as_real(planes.grad).reshape(-1, 2)
            for idx, w in corners:
                d_grid.index_add_(0, idx.reshape(-1), w.reshape(-1, 1) * g)
    out = {"loss": loss, "d_wxyz": leaf["q"].grad, "d_offset": leaf["off"].grad, "d_defocus": leaf["df"].grad}
    out = {k: v.detach().cpu().numpy() for k, v in out.items()}
    if case["volume_gradient"]:
        out["d_grid"] = torch.view_as_complex(d_grid).reshape(n, n, n)
    return out


def _exact_search(case, seed):
    real, p, observed = _search_inputs(case, seed)
    py, n = case["box"], 2 * case["box"]
    grid = _fourier64(real, n)
    table = _orientations(case)
    count = case["images"]
    w = torch.full((py // 2 + 1,), 2.0, dtype=torch.float64, device=DEV)
    w[0] = 1.0
    if py % 2 == 0:
        w[-1] = 1.0
    weight = w.expand(py, -1).clone()
    weight[0, 0] = 0.0
    obs = torch.fft.rfft2(torch.fft.ifftshift(observed.double(), dim=(-2, -1)))
    # what contrast transfer and translation do to a unit spectrum
    qx = torch.fft.rfftfreq(py, PIXEL, device=DEV, dtype=torch.float64)[None, None]
    qy = torch.fft.fftfreq(py, PIXEL, device=DEV, dtype=torch.float64)[None, :, None]
    sl = slice(0, count)
    ctf = torch.sin(2.0 * math.pi * _chi_cycles(p, sl, qx, qy) - math.atan(AC / math.sqrt(1.0 - AC * AC)))
    off = torch.as_tensor(p["off"], device=DEV)
    ph = -2.0 * math.pi * (qx * off[:, 0, None, None] + qy * off[:, 1, None, None])
    mult = torch.complex(torch.cos(ph), torch.sin(ph)) * ctf
    if py % 2 == 0:
        mult[:, py // 2, 0] = mult[:, 0, -1] = mult[:, py // 2, -1] = 0.0
    a = (weight * torch.conj(mult) * obs).reshape(count, -1)
    z = (weight * mult.abs() ** 2).reshape(count, -1)
    oo = (weight * obs.abs() ** 2).sum(dim=(-2, -1))
    best = torch.full((count,), -2.0, dtype=torch.float64, device=DEV)
    step = max(1, int(2.5e7 // (n * n)))
    for s in range(0, len(table), step):
        rot = _rotation64(torch.as_tensor(table[s:s + step], device=DEV))
        t = torch.fft.rfft2(_crop64(_irfft2(_sample64(grid, rot, n, "slice"), n), py, (-2, -1)))
        t = t.reshape(t.shape[0], -1)
        num = a.real @ t.real.T + a.imag @ t.imag.T
        den = torch.sqrt((z @ (t.abs() ** 2).T) * oo[:, None])
        best = torch.maximum(best, (num / den).max(dim=1).values)
    return {"orientation": None, "score": best.cpu().numpy()}


def _exact_network(case, seed):
    params, x, labels, near = _network_inputs(case, seed)
    layers, _ = _layers(case["size"], case["classes"])
    p = torch.as_tensor(params, device=DEV).double().requires_grad_(True)
    b = case["images"]
    a = x.double()[:, None]
    for L in layers:
        w = p[L["at"]:L["at"] + L["k"] * L["cout"]].reshape(L["k"], L["cout"])
        bias = p[L["at"] + L["k"] * L["cout"]:L["at"] + (L["k"] + 1) * L["cout"]]
        if L["pixels"] > 1 or L["k"] == 9 * L["cin"]:  # rows of w are (ky, kx, channel)
            kern = w.reshape(3, 3, L["cin"], L["cout"]).permute(3, 2, 0, 1)
            a = torch.relu(torch.nn.functional.conv2d(a, kern, bias, stride=2, padding=1))
            continue
        if a.dim() == 4:
            a = a.permute(0, 2, 3, 1).reshape(b, -1)
        a = a @ w + bias
        if L is not layers[-1]:
            a = torch.relu(a)
    t = torch.zeros((b, case["classes"]), dtype=torch.float64, device=DEV)
    rows = torch.arange(b, device=DEV)
    t[rows, labels.long()] += 0.8
    t.index_put_((rows[:, None].expand(-1, 8), near[labels.long()].long()),
                 torch.full((b, 8), 0.2 / 8, dtype=torch.float64, device=DEV), accumulate=True)
    loss = -(t * torch.log_softmax(a, dim=1)).sum(dim=1)
    loss.mean().backward()
    return {"logits": a.detach(), "loss": loss.detach(), "gradient": p.grad}


def exact(case, seed):
    k = case["kind"]
    if k == "simulate":
        return _exact_simulate(case, seed)
    if k == "batched":
        return [_images64(_fourier64(real, 2 * b), p, s) for (real, p), b, s in
                zip(_batched_inputs(case, seed), _ints(case["boxes"]), _ints(case["shapes"]))]
    if k == "gradient":
        return _exact_gradient(case, seed)
    if k == "search":
        return _exact_search(case, seed)
    return _exact_network(case, seed)
