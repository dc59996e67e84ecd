"""Performance cases: the registrations, training step and batches that a user of this package runs.

Each case is one call (or one short sequence of calls) of the public API on synthetic speckle: the images are
band-limited noise, the targets the same texture resampled under a smooth displacement field with fresh camera noise.
Kinds of case and what they stand for:

  frame     ICGNWGPU.register on a host frame: single-scale registration against a fixed reference
  pair      ICGNWGPU.set_reference + register on host images: consecutive pairs, the reference rebuilt each time
  resident  the same with both images in GPU memory (set_reference_device + register_device)
  stream    ICGNWGPUFullPyramid.register_stream on host frames: a camera sequence, uploads overlapped
  pyramid   ICGNWGPUFullPyramid.register_device on frames in GPU memory, temporal seeding with velocity
  batch     ICGNBatch.register: several pairs of uneven size, subset size and shape function in one step
  learned   LearnedSeeder.register_device: network and phase-correlation seeding of a large motion
  train     one optimisation step of the seed network (patches, forward, backward, Adam)

Sizes are those of the package's benchmark and tests (512 x 512 at subset 21 / step 10, 3840 x 2160 at 31 / 8 and
41 / 10, batches of 640 x 480 to 1920 x 1080 with subsets 15 to 41) and common camera formats with ragged edges.
"""

from __future__ import annotations

import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = str(Path(__file__).resolve().parents[1] / "live-dic_gb300")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from live_dic_gb300 import ICGNBatch, ICGNWGPU, ICGNWGPUFullPyramid, learned  # noqa: E402

DEVICE = "cuda"
_PIXEL_FLOPS = {"affine": 90.0, "translation": 80.0, "quadratic": 120.0}
_UPDATE_FLOPS = {"affine": 150.0, "translation": 60.0, "quadratic": 900.0}


def _frame(name, kind, width, height, subset, stride, **more):
    case = {"name": name, "kind": kind, "width": width, "height": height, "subset": subset, "stride": stride,
            "model": "affine", "interpolation": "bspline", "weighting": "uniform", "policy": "replace", "median": 3,
            "roi": "none", "shift": 0.6, "strain": 0.002, "wave": 0.5, "tolerance": 1e-3}
    case.update(more)
    return case


def listed():
    return [
        # The engine's defaults on a small region: the shortest call, launches and latency count.
        _frame("frame-256-default", "frame", 256, 256, 16, 16),
        # Plain affine registration of one 512 x 512 pair.
        _frame("frame-512-s21", "frame", 512, 512, 21, 10, policy="disabled", tolerance=1e-4),
        # Rigid motion tracked on raw bytes with a 5 x 5 median of the field.
        _frame("frame-1000x701-translation", "frame", 1000, 701, 15, 7, model="translation", interpolation="linear",
               policy="median", median=5, strain=0.0, wave=0.0, shift=1.4),
        # A masked specimen: Gaussian weights, windows cut by the mask's edge solved on their visible part.
        _frame("frame-1279x717-gauss-roi", "frame", 1279, 717, 25, 12, weighting="gaussian", roi="partial"),
        # A full UHD frame without seeds, and its final correlation map.
        _frame("frame-uhd-zncc", "frame", 3840, 2160, 31, 8, zncc=True, strain=0.0005),
        # Consecutive-pair mode on 720p: the reference is rebuilt for every pair.
        _frame("pair-720p-affine", "pair", 1280, 720, 21, 7, strain=0.004),
        # Consecutive pairs at UHD with the 12-parameter shape function, both images resident.
        _frame("resident-uhd-quadratic", "resident", 3840, 2160, 41, 10, model="quadratic", strain=0.001, wave=2.0),
        # The headline sequence: plate with a hole, 3-level pyramid, integer search on the first frame, temporal
        # seeding with velocity afterwards, frames resident.
        _frame("pyramid-uhd-plate", "pyramid", 3840, 2160, 31, 8, levels=3, frames=4, roi="hole", strain=0.001,
               wave=1.0),
        # A camera sequence with a large rigid motion found by phase correlation, host frames.
        _frame("stream-1080p-fourier", "stream", 1920, 1080, 31, 8, levels=2, frames=3, shift=11.0, strain=0.001),
        # Uneven pairs in one step.
        {"name": "batch-uneven", "kind": "batch", "jobs": 8, "largest": 1920, "shift": 0.8, "wave": 1.0},
        # Large motion at UHD seeded by phase correlation and the network on every 16th subset.
        _frame("learned-uhd", "learned", 3840, 2160, 31, 8, lattice=16, shift=18.0, strain=0.0006, tolerance=5e-3),
        # One training step of the seed network.
        {"name": "train-512", "kind": "train", "batch": 512, "size": 320},
    ]


def draw(rng: random.Random):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("frame", "frame", "frame", "pair", "resident", "pyramid", "stream", "batch", "learned", "train"))
    if kind == "train":
        return {"kind": kind, "batch": 128 * rng.randint(1, 4), "size": 2 * rng.randint(100, 200)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(2, 7), "largest": rng.choice((640, 1280, 1920)),
                "shift": round(rng.uniform(0.1, 1.2), 3), "wave": round(rng.uniform(0.2, 1.5), 3)}
    low = {"frame": 200, "pair": 200, "resident": 300, "pyramid": 500, "stream": 700, "learned": 1100}[kind]
    width = log_int(low, {"stream": 2000, "resident": 2600}.get(kind, 3600))
    height = min(2160, max(low * 2 // 3, int(width * rng.uniform(0.5, 0.9))))
    subset = rng.choice((15, 16, 21, 24, 25, 31, 33, 41))
    stride = max(subset // rng.choice((1, 2, 3, 4)), 5)
    more = {"shift": round(rng.uniform(0.05, 1.2), 3), "strain": round(rng.uniform(0.0, min(0.01, 6.0 / width)), 5),
            "wave": round(rng.uniform(0.0, 1.0), 3), "tolerance": rng.choice((1e-3, 1e-3, 1e-4))}
    if kind in ("frame", "pair"):
        more["interpolation"] = rng.choice(("bspline", "bspline", "bspline", "linear", "cubic"))
        more["model"] = rng.choice(("affine", "affine", "translation", "quadratic" if width < 2000 else "affine"))
        more["weighting"] = rng.choice(("uniform", "uniform", "gaussian"))
        more["policy"] = rng.choice(("replace", "flag", "disabled", "median"))
        if more["policy"] == "median":
            more["median"] = rng.choice((3, 5, 7))
        if more["model"] == "translation":
            more["strain"] = more["wave"] = 0.0
        elif kind == "frame" and more["model"] == "affine" and rng.random() < 0.4:
            more["roi"] = rng.choice(("rect", "hole"))
    elif kind == "resident":
        more["model"] = rng.choice(("affine", "quadratic"))
    elif kind in ("pyramid", "stream"):
        subset = rng.choice((21, 25, 31))
        stride = max(subset // rng.choice((2, 3, 4)), 6)
        more.update(levels=rng.choice((2, 3)), frames=rng.randint(2, 3), strain=round(rng.uniform(0.0, 0.002), 5))
        if kind == "stream":
            more["shift"] = round(rng.uniform(4.0, 14.0), 2)
        else:
            more["roi"] = rng.choice(("none", "hole"))
    elif kind == "learned":
        subset, stride = 31, rng.choice((8, 10))
        more.update(lattice=rng.choice((8, 16)), shift=round(rng.uniform(8.0, 24.0), 2),
                    strain=round(rng.uniform(0.0, 0.001), 5), tolerance=5e-3)
    if more.get("model") == "quadratic":
        stride, more["tolerance"] = max(stride, subset // 3), 1e-3
    case = _frame("", kind, width, height, subset, stride, **more)
    del case["name"]
    return case


# ---------------------------------------------------------------- images
def _generator(seed, salt):
    g = torch.Generator(device=DEVICE)
    g.manual_seed((seed * 1000003 + salt) % (1 << 62))
    return g


def _blur(image, sigma):
    r = int(math.ceil(4 * sigma))
    x = torch.arange(-r, r + 1, device=DEVICE, dtype=torch.float32)
    k = torch.exp(-0.5 * (x / sigma) ** 2)
    k = k / k.sum()
    image = torch.nn.functional.conv2d(image[None, None], k.view(1, 1, 1, -1), padding=(0, r))
    return torch.nn.functional.conv2d(image, k.view(1, 1, -1, 1), padding=(r, 0))[0, 0]


def _texture(width, height, g, margin=48):
    """Float speckle with a margin, scaled to about [20, 235]."""
    noise = torch.randn(height + 2 * margin, width + 2 * margin, device=DEVICE, generator=g)
    t = _blur(noise, 1.9)
    return (127.5 + 42.0 * t / t.std()).clamp(20.0, 235.0)


def _quantise(image, g):
    noisy = image + 0.5 * torch.randn(image.shape, device=DEVICE, generator=g)
    return noisy.round().clamp(0, 255).to(torch.uint8)


class _Field:
    """u = shift + strain, shear and one long wave about the image's centre; `load` scales it."""

    def __init__(self, case, seed, width, height):
        rng = random.Random(seed * 7919 + 17)
        angle = rng.uniform(0.0, 2.0 * math.pi)
        self.tx, self.ty = case["shift"] * math.cos(angle), case["shift"] * math.sin(angle)
        s = case.get("strain", 0.0)
        self.g = [s * rng.uniform(0.5, 1.0) * rng.choice((-1, 1)) for _ in range(4)]
        self.wave, self.length = case.get("wave", 0.0), max(400.0, 0.4 * max(width, height))
        self.phase = [rng.uniform(0.0, 2.0 * math.pi) for _ in range(2)]
        self.cx, self.cy = 0.5 * (width - 1), 0.5 * (height - 1)

    def __call__(self, x, y, load):
        dx, dy, k = x - self.cx, y - self.cy, 2.0 * math.pi / self.length
        u = self.tx + self.g[0] * dx + self.g[1] * dy + self.wave * torch.sin(k * x + self.phase[0]) * torch.cos(0.7 * k * y)
        v = self.ty + self.g[2] * dx + self.g[3] * dy + 0.7 * self.wave * torch.cos(k * x + self.phase[1])
        return load * u, load * v


def _deform(texture, field, width, height, load, g, margin=48):
    """The texture at X where x = X + u(X), bicubic, with noise."""
    y, x = torch.meshgrid(torch.arange(height, device=DEVICE, dtype=torch.float32),
                          torch.arange(width, device=DEVICE, dtype=torch.float32), indexing="ij")
    X, Y = x, y
    for _ in range(5):
        u, v = field(X, Y, load)
        X, Y = x - u, y - v
    th, tw = texture.shape
    grid = torch.stack([(X + margin) * (2.0 / (tw - 1)) - 1.0, (Y + margin) * (2.0 / (th - 1)) - 1.0], -1)
    out = torch.nn.functional.grid_sample(texture[None, None], grid[None], mode="bicubic", padding_mode="border",
                                          align_corners=True)[0, 0]
    return _quantise(out, g)


def _images(case, seed, frames=1, salt=0):
    """(reference, [targets]) on the GPU; target k carries load (k + 1 + offset) / (frames + offset)."""
    width, height = case["width"], case["height"]
    g = _generator(seed, salt)
    texture = _texture(width, height, g)
    reference = _quantise(texture[48:48 + height, 48:48 + width], g)
    field = _Field(case, seed + salt, width, height)
    offset = 6  # a sequence's frames are the last ones of a ramp
    return reference, [_deform(texture, field, width, height, (k + 1 + offset) / (frames + offset), g)
                       for k in range(frames)]


def _mask(case, seed):
    width, height, kind = case["width"], case["height"], case["roi"]
    if kind == "none":
        return None
    y, x = np.ogrid[:height, :width]
    rng = random.Random(seed * 31 + 5)
    if kind == "hole":
        r = 0.14 * min(width, height)
        return (x - 0.5 * width) ** 2 + (y - 0.5 * height) ** 2 >= r * r
    mx, my = int(width * rng.uniform(0.03, 0.08)), int(height * rng.uniform(0.03, 0.08))
    mask = np.zeros((height, width), dtype=bool)
    mask[my:height - my, mx:width - mx] = True
    r = 0.1 * min(width, height)
    mask &= (x - width * rng.uniform(0.35, 0.65)) ** 2 + (y - height * rng.uniform(0.35, 0.65)) ** 2 >= r * r
    return mask


def _grid(case):
    s, t = case["subset"], case["stride"]
    return 1 + (case["width"] - s) // t, 1 + (case["height"] - s) // t


_streams: list = []


def _stream():
    """The program's one stream for resident frames."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


# ---------------------------------------------------------------- preparation
def _engine(case):
    return ICGNWGPU(motion_model=case["model"], interpolation=case["interpolation"],
                    spatial_weighting=case["weighting"], subset_size=case["subset"], subset_stride=case["stride"],
                    outlier_policy=case["policy"], median_filter_size=case["median"])


def _prepare_frame(case, seed):
    reference, (target,) = _images(case, seed)
    engine = _engine(case)
    mask = _mask(case, seed)
    engine.set_reference(reference.cpu().numpy(), tolerance=case["tolerance"], roi_mask=mask,
                         roi_policy="partial" if case["roi"] == "partial" else "full")
    return {"kind": "frame", "engine": engine, "target": target.cpu().numpy(), "zncc": bool(case.get("zncc"))}


def _prepare_pair(case, seed):
    reference, (target,) = _images(case, seed)
    return {"kind": "pair", "engine": _engine(case), "reference": reference.cpu().numpy(),
            "target": target.cpu().numpy(), "tolerance": case["tolerance"], "mask": _mask(case, seed)}


def _prepare_resident(case, seed):
    reference, (target,) = _images(case, seed)
    gw, gh = _grid(case)
    stride = 16 if case["model"] == "quadratic" else 8
    return {"kind": "resident", "engine": _engine(case), "reference": reference, "target": target,
            "tolerance": case["tolerance"], "state": torch.zeros(gh, gw, stride, device=DEVICE), "stream": _stream()}


def _prepare_pyramid(case, seed):
    reference, targets = _images(case, seed, case["frames"])
    resident = case["kind"] == "pyramid"
    start = ({"initialization": "temporal", "temporal_prediction": "velocity", "seed_search_radius": 4} if resident
             else {"initialization": "fourier"})
    engine = ICGNWGPUFullPyramid(pyramid_levels=case["levels"], subset_size=case["subset"],
                                 subset_stride=case["stride"], **start)
    engine.set_reference(reference.cpu().numpy(), roi_mask=_mask(case, seed))
    if not resident:
        return {"kind": "stream", "engine": engine, "targets": [t.cpu().numpy() for t in targets]}
    gw, gh = _grid(case)
    return {"kind": "pyramid", "engine": engine, "targets": targets, "stream": _stream(),
            "states": [torch.zeros(gh, gw, 8, device=DEVICE) for _ in targets]}


_BATCH_SIZES = ((640, 480), (1280, 720), (1920, 1080))


def _batch_jobs(case):
    """Sizes, subsets and shape functions of the jobs, the same for every seed."""
    sizes = [s for s in _BATCH_SIZES if s[0] <= case["largest"]]
    jobs = []
    for k in range(case["jobs"]):
        w, h = sizes[k % len(sizes)]
        s = (21, 31, 15, 41)[k % 4]
        jobs.append({"width": w, "height": h, "subset": s, "stride": s // 3,
                     "model": "quadratic" if k % 3 == 1 else "affine", "roi": "rect" if k % 3 == 2 else "none",
                     "shift": case["shift"], "strain": 0.001, "wave": case["wave"]})
    return jobs


def _prepare_batch(case, seed):
    batch, targets = ICGNBatch(), []
    for k, job in enumerate(_batch_jobs(case)):
        reference, (target,) = _images(job, seed, salt=k)
        batch.add(reference.cpu().numpy(), motion_model=job["model"], subset_size=job["subset"],
                  subset_stride=job["stride"], roi_mask=_mask(job, seed + k))
        targets.append(target.cpu().numpy())
    return {"kind": "batch", "batch": batch, "targets": targets}


def _prepare_learned(case, seed):
    """The network's proposals are kept small (a scaled output layer): the global motion comes from the phase
    correlation and the node solve refines it, as for a trained network, whatever the weights."""
    reference, (target,) = _images(case, seed)
    host = reference.cpu().numpy()
    engine = _engine(case)
    engine.set_reference(host, iterations=16, tolerance=case["tolerance"])
    net = learned.SeedNet(batch=128, seed=3)
    state = net.state_dict()
    state["w6"] = state["w6"] * 0.02
    net.load_state_dict(state)
    seeder = learned.LearnedSeeder(engine, net, step=case["lattice"])
    seeder.set_reference_image(host)
    return {"kind": "learned", "seeder": seeder, "engine": engine, "target": target}


def _train_inputs(case, seed):
    size, batch = case["size"], case["batch"]
    g = _generator(seed, 0)
    texture = _texture(size, size, g)
    references, targets = [], []
    for k in range(8):
        references.append(_quantise(texture[48:48 + size, 48:48 + size], g))
        field = _Field({"shift": 6.0, "strain": 0.03, "wave": 0.0}, seed + k, size, size)
        targets.append(_deform(texture, field, size, size, 1.0, g))
    references, targets = torch.stack(references), torch.stack(targets)
    index = torch.randint(0, 8, (batch,), device=DEVICE, generator=g, dtype=torch.int32)
    centres = 32.0 + (size - 64.0) * torch.rand(batch, 2, device=DEVICE, generator=g)
    labels = torch.randn(batch, 6, device=DEVICE, generator=g)
    return references, targets, index, centres, labels


def _prepare_train(case, seed):
    references, targets, index, centres, labels = _train_inputs(case, seed)
    net = learned.SeedNet(batch=case["batch"], seed=5)

    def pointers(t):
        return torch.tensor([x.data_ptr() for x in t], dtype=torch.int64, device=DEVICE)

    return {"kind": "train", "net": net, "references": references, "targets": targets, "ref_ptrs": pointers(references),
            "tgt_ptrs": pointers(targets), "index": index, "centres": centres, "labels": labels, "size": case["size"]}


_PREPARE = {"frame": _prepare_frame, "pair": _prepare_pair, "resident": _prepare_resident, "pyramid": _prepare_pyramid,
            "stream": _prepare_pyramid, "batch": _prepare_batch, "learned": _prepare_learned, "train": _prepare_train}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------- passes
def _fields(result):
    return [result.parameters, result.status, result.iterations]


def run(state):
    kind = state["kind"]
    if kind == "frame":
        result = state["engine"].register(state["target"], include_zncc=state["zncc"])
        return _fields(result) + ([result.zncc] if state["zncc"] else [])
    if kind == "pair":
        info = state["engine"].set_reference(state["reference"], tolerance=state["tolerance"], roi_mask=state["mask"])
        return _fields(state["engine"].register(state["target"])) + [info.reference_valid]
    if kind == "resident":
        engine, reference = state["engine"], state["reference"]
        height, width = reference.shape
        engine.set_reference_device(reference.data_ptr(), width, height, tolerance=state["tolerance"])
        engine.register_device(state["target"].data_ptr(), state["state"].data_ptr(),
                               stream=state["stream"].cuda_stream)
        return [state["state"]]
    if kind == "pyramid":
        engine = state["engine"]
        engine.reset_temporal_state()
        for frame, out in zip(state["targets"], state["states"]):
            engine.register_device(frame.data_ptr(), out.data_ptr(), stream=state["stream"].cuda_stream)
        return state["states"]
    if kind == "stream":
        return [_fields(r) for r in state["engine"].register_stream(state["targets"])]
    if kind == "batch":
        return [_fields(r) for r in state["batch"].register(state["targets"])]
    if kind == "learned":
        seeder = state["seeder"]
        seeder.register_device(state["target"], counts=False)
        return [seeder.state.view(seeder.gh, seeder.gw, 8)]
    net = state["net"]
    net.load_patches(state["ref_ptrs"], state["tgt_ptrs"], state["index"], state["centres"], net.B, state["size"],
                     state["size"])
    net.forward()
    net.loss_and_grad(state["labels"])
    net.backward()
    net.adam_step(1e-3)
    return [net.out[:, :6], net.loss, net.grads, net.params]


# ---------------------------------------------------------------- work
def _solve_work(case, frames, iterations):
    gw, gh = _grid(case)
    count, model = gw * gh, case["model"]
    pixels = case["width"] * case["height"]
    per = _PIXEL_FLOPS[model] * case["subset"] ** 2 + _UPDATE_FLOPS[model]
    n = 12 if model == "quadratic" else 6
    state = 64 if model == "quadratic" else 32
    # per frame: the target's bytes, the prepared reference (three floats a pixel, metadata and inverse Hessian a
    # window) and the field written
    return {"bytes": float(frames * (pixels * 13 + count * (4 * n * n + 4 * (2 * n + 4) + state))),
            "flops": float(frames * count * per * iterations)}


def work(case):
    kind = case["kind"]
    if kind == "train":
        shapes, side, flops, weights = ((2, 32), (32, 64), (64, 128), (128, 128), (128, 64)), 64, 0.0, 0
        for k, (cin, cout) in enumerate(shapes):
            side //= 2
            flops += 2.0 * side * side * 9 * cin * cout * (2 if k == 0 else 3)
            weights += 9 * cin * cout + cout
        return {"bytes": float(case["batch"] * 4096 * 2 + 7 * 4 * weights), "flops": case["batch"] * flops}
    if kind == "batch":
        parts = [_solve_work(job, 1, 4.0) for job in _batch_jobs(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    frames = case.get("frames", 1)
    iterations = {"pyramid": 2.2, "stream": 2.2, "learned": 2.1}.get(kind, 4.0)
    got = _solve_work(case, frames, iterations)
    if kind in ("pair", "resident"):
        got["bytes"] += float(case["width"] * case["height"])
    return got


# ---------------------------------------------------------------- values in 64 bits
def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if (case["kind"] == "frame" and case["policy"] == "disabled" and case["roi"] == "none"
            and case["model"] == "affine" and case["interpolation"] == "bspline" and case["weighting"] == "uniform"
            and case["width"] * case["height"] <= 1 << 20):
        return [_exact_affine(case, seed), None, None]
    return None


def _reflect(n, pad):
    i = torch.arange(-pad, n + pad, device=DEVICE).abs()
    return torch.where(i >= n, 2 * n - 2 - i, i)


def _separable(image, taps):
    pad = len(taps) // 2
    for axis in (1, 0):
        n = image.shape[axis]
        padded = image.index_select(axis, _reflect(n, pad))
        image = sum(t * padded.narrow(axis, k, n) for k, t in enumerate(taps))
    return image


def _exact_affine(case, seed):
    """Inverse-compositional Gauss-Newton of every window in 64 bits: sigma-one Gaussian and cubic B-spline of both
    images, ZNSSD criterion, the engine's stopping rule."""
    reference, (target,) = _images(case, seed)
    S, st, W, H = case["subset"], case["stride"], case["width"], case["height"]
    gauss = np.exp(-0.5 * np.arange(-3.0, 4.0) ** 2)
    gauss = (gauss / gauss.sum()).tolist()
    pole = math.sqrt(3.0) - 2.0
    inverse = [math.sqrt(3.0) * pole ** abs(k) for k in range(-24, 25)]
    f = _separable(reference.double(), gauss)
    cf = _separable(f, inverse)
    cg = _separable(_separable(target.double(), gauss), inverse)
    side, deriv = [1 / 6, 4 / 6, 1 / 6], [-0.5, 0.0, 0.5]

    def along(image, tx, ty):
        px = image.index_select(1, _reflect(W, 1))
        image = sum(t * px.narrow(1, k, W) for k, t in enumerate(tx))
        py = image.index_select(0, _reflect(H, 1))
        return sum(t * py.narrow(0, k, H) for k, t in enumerate(ty))

    gx, gy = along(cf, deriv, side), along(cf, side, deriv)
    gw, gh = _grid(case)

    def windows(p):
        return p.unfold(0, S, st).unfold(1, S, st)[:gh, :gw].reshape(gw * gh, S * S)

    c = torch.arange(S, device=DEVICE, dtype=torch.float64) - 0.5 * (S - 1)
    ly, lx = (t.reshape(-1) for t in torch.meshgrid(c, c, indexing="ij"))
    fw, wx, wy = windows(f), windows(gx), windows(gy)
    J = torch.stack([wx, wx * lx, wx * ly, wy, wy * lx, wy * ly], -1)
    hess = torch.linalg.inv(J.transpose(1, 2) @ J)
    fm = fw - fw.mean(1, keepdim=True)
    norm_f = fm.norm(dim=1)
    jtf, sj = (J * fm[..., None]).sum(1), J.sum(1)
    n = gw * gh
    yy, xx = torch.meshgrid(torch.arange(gh, device=DEVICE), torch.arange(gw, device=DEVICE), indexing="ij")
    ox, oy = (xx.reshape(-1, 1) * st + 0.5 * (S - 1)).double(), (yy.reshape(-1, 1) * st + 0.5 * (S - 1)).double()
    p = torch.zeros(n, 6, device=DEVICE, dtype=torch.float64)
    live = torch.ones(n, device=DEVICE, dtype=torch.bool)
    half = 0.5 * (S - 1)
    corners = torch.tensor([[-half, -half], [half, -half], [-half, half], [half, half]], device=DEVICE,
                           dtype=torch.float64)
    flat = cg.reshape(-1)

    def place(p, x, y):
        return (ox + x + p[:, 0:1] + p[:, 1:2] * x + p[:, 2:3] * y, oy + y + p[:, 3:4] + p[:, 4:5] * x + p[:, 5:6] * y)

    def weights(t):
        s = 1.0 - t
        return (s ** 3 / 6, (3 * t ** 3 - 6 * t ** 2 + 4) / 6, (-3 * t ** 3 + 3 * t ** 2 + 3 * t + 1) / 6, t ** 3 / 6)

    for _ in range(30):
        cx, cy = place(p, corners[:, 0], corners[:, 1])
        inside = ((cx >= 2) & (cy >= 2) & (cx <= W - 3) & (cy <= H - 3)).all(1)
        live = live & inside
        if not bool(live.any()):
            break
        X, Y = place(p, lx, ly)
        bx, by = X.floor(), Y.floor()
        wX, wY = weights(X - bx), weights(Y - by)
        bx, by = bx.long().clamp(1, W - 3), by.long().clamp(1, H - 3)
        g = sum(wY[j] * sum(wX[i] * flat[(by + j - 1) * W + bx + i - 1] for i in range(4)) for j in range(4))
        gm = g.mean(1, keepdim=True)
        norm_g = (g - gm).norm(dim=1)
        r = jtf - (norm_f / norm_g)[:, None] * ((J * g[..., None]).sum(1) - gm * sj)
        d = -(hess @ r[..., None])[..., 0]
        a = torch.linalg.inv(torch.stack([1 + d[:, 1], d[:, 2], d[:, 4], 1 + d[:, 5]], -1).view(n, 2, 2))
        w = torch.stack([1 + p[:, 1], p[:, 2], p[:, 4], 1 + p[:, 5]], -1).view(n, 2, 2)
        t = p[:, [0, 3]] - (w @ (a @ d[:, [0, 3]][..., None]))[..., 0]
        w = w @ a
        new = torch.stack([t[:, 0], w[:, 0, 0] - 1, w[:, 0, 1], t[:, 1], w[:, 1, 0], w[:, 1, 1] - 1], -1)
        p = torch.where(live[:, None], new, p)
        moved = torch.hypot(d[:, 0:1] + d[:, 1:2] * corners[:, 0] + d[:, 2:3] * corners[:, 1],
                            d[:, 3:4] + d[:, 4:5] * corners[:, 0] + d[:, 5:6] * corners[:, 1]).amax(1)
        live = live & (moved >= case["tolerance"])
    return p.view(gh, gw, 6)


def _exact_train(case, seed):
    """The same step in 64 bits through autograd, from the same initial weights."""
    references, targets, index, centres, labels = _train_inputs(case, seed)
    batch, size = case["batch"], case["size"]
    x0 = torch.floor(centres + 0.5).long() - 32
    span = torch.arange(64, device=DEVICE)
    rows = (x0[:, 1:2] + span).clamp(0, size - 1)
    cols = (x0[:, 0:1] + span).clamp(0, size - 1)
    pick = index.long()[:, None, None], rows[:, :, None], cols[:, None, :]
    patches = []
    for images in (references, targets):
        v = images[pick].double()
        mean = v.mean((1, 2), keepdim=True)
        var = (v * v).mean((1, 2), keepdim=True) - mean * mean
        patches.append((v - mean) * var.clamp(min=1e-2).rsqrt())
    x = torch.stack(patches, 1)
    g = torch.Generator(device="cpu").manual_seed(5)
    params = []
    for cin, cout in learned.CONV_CHANNELS:
        kp = (9 * cin + 63) // 64 * 64
        w = torch.zeros(cout, kp)
        w[:, :9 * cin] = torch.randn(cout, 9 * cin, generator=g) * math.sqrt(2.0 / (9 * cin))
        params.append(w.to(DEVICE).double().requires_grad_())
    params += [torch.zeros(cout, device=DEVICE, dtype=torch.float64, requires_grad=True)
               for _, cout in learned.CONV_CHANNELS]
    w6 = torch.zeros(16, 256)
    w6[:6] = torch.randn(6, 256, generator=g) * math.sqrt(1.0 / 256)
    params.append(w6.to(DEVICE).double().requires_grad_())
    params.append(torch.zeros(16, device=DEVICE, dtype=torch.float64, requires_grad=True))
    for k, (cin, cout) in enumerate(learned.CONV_CHANNELS):
        kernel = params[k][:, :9 * cin].view(cout, 3, 3, cin).permute(0, 3, 1, 2)
        x = torch.relu(_convolve(x, kernel) + params[5 + k].view(1, -1, 1, 1))
    out = x.permute(0, 2, 3, 1).reshape(batch, -1) @ params[10].T + params[11]
    loss = 0.5 * (out[:, :6] - labels.double()).square().sum() / batch
    loss.backward()
    grads = [p.grad for p in params]
    with torch.no_grad():
        # Adam's first step is the gradient's sign times the rate: for biases, which start at zero, that is the whole
        # value, and the sign of a gradient near zero is not determined by BF16 products.
        updated = [None if 5 <= k <= 9 else p - 1e-3 * d / (d.abs() + 1e-8)
                   for k, (p, d) in enumerate(zip(params, grads))]
    return [out[:, :6].detach(), loss.detach().view(1), grads, updated]


def _convolve(x, kernel):
    """3 x 3, stride 2, pad 1, as nine matrix products in 64 bits."""
    side = x.shape[-1] // 2
    padded = torch.nn.functional.pad(x, (1, 1, 1, 1))
    return sum(torch.einsum("bcyx,oc->boyx", padded[:, :, ky:ky + 2 * side:2, kx:kx + 2 * side:2], kernel[:, :, ky, kx])
               for ky in range(3) for kx in range(3))
