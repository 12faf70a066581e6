"""The calls that a program using this library makes, as cases to time.

Deconvolution of 3-D microscopy volumes is what the library is for, so most
cases are whole solves through ``clarity_b200.api``: a volume and a PSF go in,
the restored volume comes out.  They span the sizes of this repository's
configurations, tests and benchmark: from the 16 x 16 x 8 test volume, whose
cost is launches, over 256 x 256 x 64, to 512 x 512 x 128, whose work box
(image + PSF per axis) holds 268 million voxels.  PSFs come at the image's own
size, as the benchmark has them, and smaller, as a program that crops its PSF
has them; the work boxes are powers of two, other even lengths and odd ones.
The learned start's network is measured by its convolution layer, forward
alone (prediction) and forward with both gradients (training).

A volume case is described by its operation, the image's and the PSF's extents
(x fastest) and the iterations; a layer case by its channels and voxels.
"""
import math

import numpy as np
import torch

from clarity_b200 import api, unet

EPSILON = 1e-3  # the Wiener filter's constant in the 256 x 256 x 64 configuration


def _volume(name, op, image, psf, iterations=0):
    return {"name": name, "op": op, "x": image[0], "y": image[1], "z": image[2],
            "kx": psf[0], "ky": psf[1], "kz": psf[2], "iterations": iterations}


def _layer(name, direction, c1, c2, cout, size):
    return {"name": name, "op": "layer", "direction": direction, "c1": c1, "c2": c2,
            "cout": cout, "x": size[0], "y": size[1], "z": size[2]}


def listed():
    return [
        # the reference's test volume: one convolution, where latency and launches count
        _volume("convolve 16x16x8", "convolve", (16, 16, 8), (16, 16, 8)),
        # a small crop deconvolved on the spot: ten iterations, launch-bound
        _volume("rl 64x64x32", "rl", (64, 64, 32), (64, 64, 32), 10),
        # one filter pass from and to ordinary host memory, as callers of the C API make it
        _volume("wiener host 256x256x64", "wiener_host", (256, 256, 64), (256, 256, 64)),
        # the benchmark's volume and PSF, enough iterations that the steady state rules
        _volume("rl 256x256x64", "rl", (256, 256, 64), (256, 256, 64), 50),
        _volume("jvc 256x256x64", "jvc", (256, 256, 64), (256, 256, 64), 20),
        # the same volume by the accelerated form, to the iteration count that meets its target
        _volume("accel 256x256x64", "accel", (256, 256, 64), (256, 256, 64), 16),
        # the largest configuration
        _volume("rl 512x512x128", "rl", (512, 512, 128), (512, 512, 128), 5),
        # a cropped PSF: the work box is no power of two
        _volume("rl 256x256x64 psf 64x64x32", "rl", (256, 256, 64), (64, 64, 32), 20),
        # a volume cut to its specimen, with an odd work box on every axis
        _volume("rl 140x126x36 psf 31x21x13", "rl", (140, 126, 36), (31, 21, 13), 20),
        # volumes of uneven sizes restored together, as the training pairs are made
        {"name": "batch of 12", "op": "batch", "count": 12, "sizes": 5, "iterations": 5},
        # the decoder's full-resolution layer on a training patch: output and all gradients
        _layer("layer train 16+32 to 16", "train", 16, 32, 16, (128, 128, 48)),
        # an encoder layer of the prediction on a 256 x 256 x 64 volume
        _layer("layer predict 32 to 32", "predict", 32, 0, 32, (128, 128, 32)),
    ]


# Voxels of the work box times iterations (one for the single-pass filters) that a drawn
# solve stays below: the 512 x 512 x 128 case's.
MOST_WORK = 1024 * 1024 * 256 * 5


def _is_smooth(n):
    """Whether n has no prime factor above 13."""
    for p in (2, 3, 5, 7, 11, 13):
        while n % p == 0:
            n //= p
    return n == 1


def _smooth(lo, hi, rng):
    """A length in [lo, hi] without large factors, spread over its logarithm."""
    while True:
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))
        if lo <= n <= hi and _is_smooth(n):
            return n


def draw(rng):
    op = rng.choice(["convolve", "wiener_host", "rl", "rl", "rl", "rl", "jvc", "accel", "batch",
                     "layer"])
    if op == "batch":
        return {"op": op, "count": rng.randint(3, 12), "sizes": rng.randrange(1000),
                "iterations": rng.randint(2, 5)}
    if op == "layer":
        c1 = rng.choice([16, 32, 64])
        c2 = rng.choice([0, 2 * c1])
        f = {16: 1, 32: 2, 64: 4}[c1]
        size = (32 * rng.randint(2, 8) // f, 16 * rng.randint(2, 16) // f,
                8 * rng.randint(2, 8) // f)
        size = tuple(8 * max(1, s // 8) for s in size)
        return _unnamed(_layer("", rng.choice(["train", "predict"]), c1, c2, c1, size))
    while True:
        # the work box is what the transforms see; the PSF takes a part of each axis.  Fields of
        # view are about square and thinner than wide.
        nx = _smooth(24, 1024, rng)
        box = (nx, _smooth(max(24, int(0.6 * nx)), min(1024, int(1.6 * nx)), rng),
               _smooth(max(12, nx // 8), max(16, min(256, int(0.6 * nx))), rng))
        same = rng.random() < 0.4
        if same:
            box = tuple(2 * (n // 2) for n in box)
            if not all(_is_smooth(n) for n in box):
                continue
        image = tuple(n // 2 if same else n - max(1, int(n * rng.uniform(0.08, 0.5))) for n in box)
        psf = tuple(n - i for n, i in zip(box, image))
        iterations = {"rl": rng.randint(2, 50), "jvc": rng.randint(2, 20),
                      "accel": rng.randint(2, 16)}.get(op, 0)
        if math.prod(box) * max(1, iterations) * (2 if op == "accel" else 1) <= MOST_WORK:
            return _unnamed(_volume("", op, image, psf, iterations))


def _unnamed(case):
    return {k: v for k, v in case.items() if k != "name"}


# ------------------------------------------------------------------- inputs
def _gaussian(shape, sigma_xy, sigma_z):
    """A separable Gaussian centred at n/2, unit sum (float64)."""
    axes = []
    for n, s in zip(shape, (sigma_z, sigma_xy, sigma_xy)):
        t = torch.arange(n, dtype=torch.float64, device="cuda") - n // 2
        axes.append(torch.exp(-0.5 * (t / s) ** 2))
    p = axes[0][:, None, None] * axes[1][None, :, None] * axes[2][None, None, :]
    return p / p.sum()


def _pair(shape, psf_shape, seed):
    """An observed volume and its PSF (float32, z-y-x, on the GPU): spheres of radius 1.5 to 4
    and whole intensities 200 to 1000 on a background of 10, at one per 7000 voxels, blurred by
    the PSF (a Gaussian core with a wide halo) and Poisson noise on top."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    nz, ny, nx = shape

    def uniform(n, lo, hi):
        return lo + (hi - lo) * torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)

    n = max(1, nz * ny * nx // 7000)
    cz, cy, cx = uniform(n, 0, nz), uniform(n, 0, ny), uniform(n, 0, nx)
    rad, amp = uniform(n, 1.5, 4.0), torch.floor(uniform(n, 200, 1000))
    d = torch.arange(-4, 5, device="cuda")
    oz, oy, ox = (a.reshape(1, -1) for a in torch.meshgrid(d, d, d, indexing="ij"))
    iz, iy, ix = (torch.floor(c).long()[:, None] + o for c, o in ((cz, oz), (cy, oy), (cx, ox)))
    inside = ((iz - cz[:, None]) ** 2 + (iy - cy[:, None]) ** 2 + (ix - cx[:, None]) ** 2
              <= rad[:, None] ** 2)
    inside &= (iz >= 0) & (iz < nz) & (iy >= 0) & (iy < ny) & (ix >= 0) & (ix < nx)
    vol = torch.full((nz * ny * nx,), 10.0, device="cuda")
    vol.index_add_(0, ((iz * ny + iy) * nx + ix)[inside],
                   amp[:, None].expand(inside.shape)[inside].float())  # whole numbers: exact sums
    vol = vol.reshape(shape)
    core = float(uniform(1, 1.2, 2.5).item())
    psf = 0.9 * _gaussian(psf_shape, core, 2.4 * core) + 0.1 * _gaussian(psf_shape, 3 * core,
                                                                        6 * core)
    psf = (psf / psf.sum()).float()
    # the blur at the volume's own extent, as the phantom generator of this package does it
    kern = torch.zeros(shape, device="cuda")
    cut = tuple(slice(max(0, k // 2 - s // 2), max(0, k // 2 - s // 2) + min(s, k))
                for s, k in zip(shape, psf_shape))
    part = psf[cut]
    kern[tuple(slice(0, m) for m in part.shape)] = part
    kern = torch.roll(kern, tuple(-(k // 2 - c.start) for k, c in zip(psf_shape, cut)), (0, 1, 2))
    blurred = torch.fft.irfftn(torch.fft.rfftn(vol) * torch.fft.rfftn(kern), s=shape).clamp_min(0)
    return torch.poisson(blurred, generator=gen).contiguous(), psf.contiguous()


def _batch_shapes(case):
    """Image extents (z, y, x) of the batched workload: x, y in 16*{6..20}, z in 8*{2..12}."""
    r = np.random.default_rng(case["sizes"])
    return [(8 * int(r.integers(2, 13)), 16 * int(r.integers(6, 21)), 16 * int(r.integers(6, 21)))
            for _ in range(case["count"])]


def _layer_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    D, H, W, c1, c2, co = (case[k] for k in ("z", "y", "x", "c1", "c2", "cout"))

    def normal(*shape, scale=1.0):
        return torch.randn(shape, generator=gen, device="cuda") * scale

    cin = c1 + c2
    s = {"x1": normal(D, H, W, c1).clamp_min(0).bfloat16(),  # what a ReLU leaves
         "x2": normal(D // 2, H // 2, W // 2, c2).clamp_min(0).bfloat16() if c2 else None,
         "b": normal(co, scale=0.1), "co": co, "train": case["direction"] == "train"}
    w = normal(co, 27, cin, scale=math.sqrt(2.0 / (27 * cin))).bfloat16()
    s["w"] = w.reshape(-1).contiguous()
    if s["train"]:
        # the backward-data weights: taps mirrored, channels exchanged
        s["wb"] = w.flip(1).permute(2, 1, 0).contiguous().reshape(-1)
        dy = normal(D, H, W, co, scale=1e-2)
        s["dy"] = (dy * (normal(D, H, W, co) > 0)).bfloat16()
        s["dw"] = torch.zeros(co * 27 * cin, device="cuda")
        s["db"] = torch.zeros(co, device="cuda")
    return s


def prepare(case, seed):
    api.load()
    if case["op"] == "layer":
        return dict(_layer_inputs(case, seed), op="layer")
    if case["op"] == "batch":
        pairs = [_pair(s, s, seed * 64 + i) for i, s in enumerate(_batch_shapes(case))]
        return {"op": "batch", "images": [p[0] for p in pairs], "psfs": [p[1] for p in pairs],
                "outs": [torch.empty_like(p[0]) for p in pairs], "n": case["iterations"]}
    image, psf = _pair((case["z"], case["y"], case["x"]), (case["kz"], case["ky"], case["kx"]),
                       seed)
    if case["op"] == "wiener_host":
        return {"op": case["op"], "image": image.cpu().numpy(), "psf": psf.cpu().numpy()}
    return {"op": case["op"], "image": image, "psf": psf, "out": torch.empty_like(image),
            "n": case["iterations"]}


# --------------------------------------------------------------------- run
def run(s):
    op = s["op"]
    if op == "layer":
        y = unet.conv3(s["x1"], s["w"], s["co"], bias=s["b"], relu=True, x2=s["x2"])
        if not s["train"]:
            return y
        cin = s["x1"].shape[3] + (s["x2"].shape[3] if s["x2"] is not None else 0)
        dx = unet.conv3(s["dy"], s["wb"], cin, relu=False)
        s["dw"].zero_()
        s["db"].zero_()
        unet.conv3_wgrad(s["x1"], s["dy"], s["dw"], s["db"], x2=s["x2"])
        return [y, dx, s["dw"], s["db"]]
    if op == "batch":
        return api.ml_batch_device(s["images"], s["psfs"], s["outs"], s["n"], graph=False)
    if op == "wiener_host":
        return api.wiener_deconvolve(s["image"], s["psf"], EPSILON)
    if op == "convolve":
        return api.convolve_device(s["image"], s["psf"], s["out"])
    if op == "rl":
        return api.ml_device(s["image"], s["psf"], s["out"], s["n"])
    if op == "jvc":
        return api.jvc_device(s["image"], s["psf"], s["out"], s["n"])
    return api.ml_accel_device(s["image"], s["psf"], s["out"], s["n"])


# -------------------------------------------------------------------- work
def _solve_work(image, psf, op, iterations):
    """Bytes: image, PSF and result once.  Operations: the real transforms of the work box that
    the method is made of (2.5 n log2 n each), the OTF's among them."""
    n = math.prod(a + b for a, b in zip(image, psf))
    transforms = {"rl": 4 * iterations, "accel": 4 * iterations, "jvc": 2 * iterations}.get(op, 2)
    return {"bytes": 4.0 * (2 * math.prod(image) + math.prod(psf)),
            "flops": (1 + transforms) * 2.5 * n * math.log2(n)}


def work(case):
    if case["op"] == "layer":
        vox, cin, co = case["x"] * case["y"] * case["z"], case["c1"] + case["c2"], case["cout"]
        one = 2.0 * vox * co * 27 * cin
        x = 2.0 * vox * (case["c1"] + case["c2"] / 8)
        if case["direction"] == "predict":
            return {"bytes": x + 2 * co * 27 * cin + 2 * vox * co, "flops": one}
        return {"bytes": x + 8 * co * 27 * cin + 2 * vox * (2 * co + cin), "flops": 3 * one}
    if case["op"] == "batch":
        each = [_solve_work(s, s, "rl", case["iterations"]) for s in _batch_shapes(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    return _solve_work((case["x"], case["y"], case["z"]), (case["kx"], case["ky"], case["kz"]),
                       case["op"], case["iterations"])


# ------------------------------------------------------------------- exact
class _Box:
    """The circular convolution on the padded work box in 64 bits."""

    def __init__(self, image, psf):
        self.shape = tuple(a + b for a, b in zip(image.shape, psf.shape))
        self.inside = tuple(slice(0, n) for n in image.shape)
        self.otf = torch.fft.rfftn(torch.roll(self.pad(psf), tuple(-(k // 2) for k in psf.shape),
                                              (0, 1, 2)))
        self.g = self.pad(image)

    def pad(self, a):
        p = torch.zeros(self.shape, dtype=torch.float64, device="cuda")
        p[tuple(slice(0, n) for n in a.shape)] = a.double()
        return p

    def blur(self, u):
        return torch.fft.irfftn(torch.fft.rfftn(u) * self.otf, s=self.shape)

    def step(self, u):
        """Richardson-Lucy: u times the blurred ratio, rescaled to the image's sum."""
        b = self.blur(u)
        r = torch.where(b.abs() < 1e-5, torch.zeros_like(b), self.g / b)
        v = u * self.blur(r)
        return v * (self.g.sum() / v.sum())


def _exact_solve(image, psf, op, iterations):
    box = _Box(image, psf)
    if op == "convolve":
        u = box.blur(box.g)
    elif op == "wiener_host":
        h = box.otf
        u = torch.fft.irfftn(torch.fft.rfftn(box.g) * h.conj() / (h.abs() ** 2 + EPSILON),
                             s=box.shape)
    elif op == "jvc":
        A = 0.5 * box.g.max()
        u = box.g
        for _ in range(max(1, iterations)):
            o = box.blur(u)
            u = (u + (1 - (o - A) ** 2 / A ** 2) * (box.g - o)).clamp_min(0)
    elif op == "rl":
        u = box.g
        for _ in range(iterations):
            u = box.step(u)
    else:
        u, before, alpha, last = box.g, box.g, 0.0, None
        for _ in range(iterations):
            y = (u + alpha * (u - before)).clamp_min(0)
            before, u = u, box.step(y)
            g = u - y
            if last is not None:
                d = float((last * last).sum())
                alpha = min(1.0, max(0.0, float((g * last).sum()) / d)) if d > 0 else 0.0
            last = g
    return u[box.inside].contiguous()


def _exact_layer(case, seed):
    s = _layer_inputs(case, seed)
    D, H, W, co = case["z"], case["y"], case["x"], case["cout"]
    x = s["x1"].double()
    if s["x2"] is not None:
        up = s["x2"].double()
        for d in range(3):
            up = up.repeat_interleave(2, d)
        x = torch.cat([x, up], 3)
    cin = x.shape[3]
    w = s["w"].double().reshape(co, 27, cin)
    taps = [(t // 9, t // 3 % 3, t % 3) for t in range(27)]

    def shifted(a):
        p = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1, 1, 1))
        for t, (i, j, k) in enumerate(taps):
            yield t, p[i:i + D, j:j + H, k:k + W].reshape(D * H * W, -1)

    y = s["b"].double().expand(D * H * W, co).clone()
    for t, a in shifted(x):
        y += a @ w[:, t].T
    y = y.clamp_min(0).reshape(D, H, W, co)
    if not s["train"]:
        return y
    dy = s["dy"].double()
    dx = torch.zeros(D * H * W, cin, dtype=torch.float64, device="cuda")
    for t, a in shifted(dy):
        dx += a @ w[:, 26 - t]
    dw = torch.zeros(co, 27, cin, dtype=torch.float64, device="cuda")
    flat = dy.reshape(-1, co)
    for t, a in shifted(x):
        dw[:, t] = flat.T @ a
    return [y, dx.reshape(D, H, W, cin), dw.reshape(-1), flat.sum(0)]


def exact(case, seed):
    if case["op"] == "layer":
        return _exact_layer(case, seed)
    if case["op"] == "batch":
        s = prepare(case, seed)
        return [_exact_solve(i, p, "rl", s["n"]) for i, p in zip(s["images"], s["psfs"])]
    image, psf = _pair((case["z"], case["y"], case["x"]), (case["kz"], case["ky"], case["kx"]),
                       seed)
    out = _exact_solve(image, psf, case["op"], case["iterations"])
    return out.cpu().numpy() if case["op"] == "wiener_host" else out
