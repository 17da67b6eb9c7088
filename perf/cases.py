"""The work whose speed counts: calls that programs make through the public
entry points, from a single field of view to a whole light-sheet stack.

A case is a dict of plain values; its "task" names the entry point:

  segment       cle.voronoi_otsu_labeling of one image
  tiles         VolBatch: voronoi_otsu_labeling over a fixed set of tiles
  measure       cle.statistics_of_labelled_pixels of a given label image
  dense         cle.gauss_otsu_labeling (connected components of the mask)
  blur          cle.gaussian_blur
  top_hat       cle.top_hat_box
  voronoi       cle.voronoi_labeling of a binary image of spots
  map           cle.label_mean_intensity_map

Images are synthetic tissue made on the GPU from the seed alone: bright
ellipsoidal cells over a slow background, with shot noise.
"""
import math

import torch

import pyclesperanto_prototype_b200 as cle
from pyclesperanto_prototype_b200 import B200Array
from pyclesperanto_prototype_b200.batch import VolBatch

DTYPES = {"uint8": torch.uint8, "uint16": torch.uint16, "float32": torch.float32, "uint32": torch.uint32}
BYTES = {"uint8": 1, "uint16": 2, "float32": 4, "uint32": 4}
CELLS_3D = 5.6e-5      # cells per voxel of a volume: the light-sheet stack's 30000 in 512 x 1024 x 1024
CELLS_2D = 9e-4        # and of an image: 60 in 256 x 256
PITCH = 24             # spacing of the cells of a label image


def listed():
    return [
        # one small field of view in an interactive session: latency
        dict(name="segment_small", task="segment", d=0, h=256, w=256, dtype="float32", spot=3.5, outline=1.0),
        # a camera frame or a slide region, 8 bits, the defaults
        dict(name="segment_slide", task="segment", d=0, h=2048, w=2048, dtype="uint8", spot=2.0, outline=2.0),
        # a confocal stack of nuclei, two different sigmas
        dict(name="segment_nuclei", task="segment", d=128, h=512, w=512, dtype="uint16", spot=2.0, outline=1.0),
        # a crop of a stack after some filter: float32, no size a round number
        dict(name="segment_odd", task="segment", d=61, h=479, w=347, dtype="float32", spot=3.5, outline=1.0),
        # a whole light-sheet stack: the largest
        dict(name="segment_lightsheet", task="segment", d=512, h=1024, w=1024, dtype="uint16", spot=2.0, outline=2.0),
        # a well plate's or a tiled stack's tiles of mixed sizes, all in one batch
        dict(name="segment_tiles", task="tiles", count=32, least=64 * 64, most=64 * 256 * 256, dtype="float32",
             spot=3.5, outline=1.0),
        # the measurements of a segmented light-sheet stack
        dict(name="measure_lightsheet", task="measure", d=512, h=1024, w=1024, dtype="uint16", labels="uint32"),
        # dense segmentation without spots
        dict(name="dense_volume", task="dense", d=128, h=1024, w=1024, dtype="uint16", outline=2.0),
        # background estimation: a wide Gaussian
        dict(name="blur_wide", task="blur", d=64, h=1024, w=1024, dtype="float32", sx=10.0, sy=10.0, sz=10.0),
        # background subtraction before a segmentation
        dict(name="top_hat_volume", task="top_hat", d=100, h=512, w=512, dtype="uint16", rx=10.0, ry=10.0, rz=10.0),
        # spots to territories over the whole image
        dict(name="voronoi_image", task="voronoi", d=0, h=1024, w=1024, dtype="uint8"),
        # a parametric map for display
        dict(name="map_image", task="map", d=0, h=2048, w=1024, dtype="float32", labels="uint32"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, least, most):
    """(d, h, w) of an image (d = 0) or a volume of about `least` to `most` voxels; every other one of round sizes."""
    n = _log_uniform(rng, least, most)
    flat = n < 1 << 15 or (n < 1 << 23 and rng.random() < 0.4)
    d = 0 if flat else int(min(512, max(8, n ** (1 / 3) * rng.uniform(0.3, 1.0))))
    area = n / max(d, 1)
    h = max(16, int(math.sqrt(area) * rng.uniform(0.7, 1.4)))
    w = max(16, int(area / h))
    if rng.random() < 0.5:
        h, w = max(16, h // 16 * 16), max(16, w // 16 * 16)
    return d, h, w


def draw(rng):
    task = rng.choice(["segment", "segment", "segment", "segment", "tiles", "measure", "measure", "dense", "blur",
                       "blur", "top_hat", "voronoi", "map"])
    if task == "tiles":
        return dict(task=task, count=rng.randint(8, 48), least=64 * 64, most=_log_uniform(rng, 256 * 256, 64 * 256 * 256),
                    dtype=rng.choice(["float32", "uint16"]), spot=rng.choice([2.0, 3.5]), outline=rng.choice([1.0, 2.0]))
    least = 1 << 12
    most = {"segment": 1 << 27, "measure": 1 << 27, "dense": 1 << 27, "blur": 1 << 26,
            "top_hat": 1 << 25, "voronoi": 1 << 23, "map": 1 << 25}[task]
    d, h, w = _size(rng, least, most)
    case = dict(task=task, d=d, h=h, w=w, dtype=rng.choice(["uint8", "uint16", "uint16", "float32"]))
    if task == "segment":
        case["spot"] = rng.choice([1.0, 1.5, 2.0, 2.0, 3.0, 3.5, 5.0])
        case["outline"] = rng.choice([1.0, 1.0, 2.0, 2.0, 3.0])
    elif task == "dense":
        case["outline"] = rng.choice([1.0, 2.0, 2.0, 3.0])
    elif task == "blur":
        s = rng.choice([1.0, 2.0, 3.0, 5.0, 10.0, round(rng.uniform(0.5, 10.0), 2)])
        case.update(sx=s, sy=s, sz=s)
        if rng.random() < 0.3:
            case["sz"] = round(s / 2, 3)         # voxels twice as deep as wide
    elif task == "top_hat":
        r = float(rng.choice([1, 3, 5, 10, 15]))
        case.update(rx=r, ry=r, rz=r if rng.random() < 0.6 else 0.0)
    elif task in ("measure", "map"):
        case["labels"] = rng.choice(["uint32", "uint32", "float32"])   # a numpy label image arrives as float32
    elif task == "voronoi":
        case["dtype"] = "uint8"
    return case


# ---- inputs -----------------------------------------------------------------
def _shape(case):
    return (case["d"], case["h"], case["w"]) if case["d"] else (case["h"], case["w"])


def _stamp(canvas, centres, axes, values):
    """Ellipsoids of `values` at integer `centres` (n x dims) with semi-axes `axes`, the largest value on overlaps."""
    shape, dims, dev = canvas.shape, canvas.dim(), canvas.device
    r = [int(math.ceil(float(a))) for a in axes.max(0).values] if len(axes) else [0] * dims
    offs = torch.stack([o.reshape(-1) for o in torch.meshgrid(
        *[torch.arange(-k, k + 1, device=dev) for k in r], indexing="ij")], 1)
    flat = canvas.view(-1)
    step = max(1, (1 << 25) // len(offs))
    for a in range(0, len(centres), step):
        c, ax, v = centres[a:a + step], axes[a:a + step], values[a:a + step]
        at = torch.zeros((len(c), len(offs)), dtype=torch.int64, device=dev)
        inside = torch.zeros((len(c), len(offs)), device=dev)
        ok = torch.ones((len(c), len(offs)), dtype=torch.bool, device=dev)
        for k in range(dims):
            p = c[:, k, None] + offs[None, :, k]
            ok &= (p >= 0) & (p < shape[k])
            at = at * shape[k] + p
            inside += (offs[None, :, k] / ax[:, k, None]) ** 2
        ok &= inside <= 1.0
        flat.scatter_reduce_(0, at[ok], v[:, None].expand_as(at)[ok], "amax")


def _image(shape, dtype, seed):
    """A tissue image: background 80 to 400 (8 to 40 in 8 bits), cells of 800 to 3000 (80 to 250), shot noise."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    img = torch.full(shape, 240.0, device="cuda")
    grid = [torch.linspace(0, 1, s, device="cuda").view([-1 if i == k else 1 for i in range(len(shape))])
            for k, s in enumerate(shape)]
    wave = torch.sin(math.pi * grid[-1] + 0.5) * torch.cos(2 * math.pi * grid[-2])
    img += 160.0 * (wave * torch.sin(2 * math.pi * grid[0] + 1.0) if len(shape) == 3 else wave)
    n = max(1, round((CELLS_3D if len(shape) == 3 else CELLS_2D) * img.numel()))
    rnd = torch.rand((n, 7), generator=g, device="cuda")
    size = torch.tensor(shape, device="cuda", dtype=torch.float32)
    centres = (rnd[:, :len(shape)] * size).long()
    _stamp(img, centres, 4 + 6 * rnd[:, 3:3 + len(shape)], 800 + 2200 * rnd[:, 6])
    if dtype == "uint8":
        img /= 12.0
    img = torch.poisson(img, generator=g)
    return img.clamp_(0, 255 if dtype == "uint8" else 65535).to(torch.int32).to(DTYPES[dtype]) \
        if dtype != "float32" else img


def _label_cells(shape, seed):
    """An int32 label image 0 .. n, every label present: cells on a jittered grid, about a quarter of the voxels."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    axes = [torch.arange(min(PITCH // 2, s // 2), s, PITCH, device="cuda") for s in shape]
    centres = torch.stack([c.reshape(-1) for c in torch.meshgrid(*axes, indexing="ij")], 1)
    n = len(centres)
    rnd = torch.rand((n, 6), generator=g, device="cuda")
    jitter = ((rnd[:, :len(shape)] - 0.5) * (PITCH / 2)).long()
    last = torch.tensor(shape, device="cuda") - 1
    centres = torch.minimum(torch.clamp(centres + jitter, min=0), last)
    order = torch.randperm(n, generator=g, device="cuda")       # labels in no order of place
    lab = torch.zeros(shape, dtype=torch.int32, device="cuda")
    _stamp(lab, centres, (PITCH / 4) * (1 + rnd[:, 3:3 + len(shape)]), (order + 1).to(torch.int32))
    return lab


def _spots(shape, seed):
    """Small bright spots as a 0 / 1 image."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = max(1, round((CELLS_3D if len(shape) == 3 else CELLS_2D) * math.prod(shape)))
    rnd = torch.rand((n, 6), generator=g, device="cuda")
    centres = (rnd[:, :len(shape)] * torch.tensor(shape, device="cuda", dtype=torch.float32)).long()
    b = torch.zeros(shape, dtype=torch.int32, device="cuda")
    _stamp(b, centres, 1 + rnd[:, 3:3 + len(shape)], torch.ones(n, dtype=torch.int32, device="cuda"))
    return b.to(torch.uint8)


def _tile_shapes(case):
    """Shapes of the tiles, the same for every seed: voxel counts log-uniform, 2D and 3D mixed."""
    got = []
    for i in range(case["count"]):
        f = (i * 0.6180339887498949) % 1.0
        n = case["least"] * (case["most"] / case["least"]) ** f
        if n < 1 << 15 or i % 4 == 0:
            n = min(n, 1 << 20)
            h = int(math.sqrt(n))
            got.append((h, max(16, int(n / h))))
        else:
            d = max(8, int((n / 16) ** (1 / 3)))
            h = int(math.sqrt(n / d))
            got.append((d, h, max(16, int(n / (d * h)))))
    return got


def prepare(case, seed):
    task, seed = case["task"], int(seed)
    if task == "tiles":
        tiles = [_image(s, case["dtype"], seed * 1000 + i) for i, s in enumerate(_tile_shapes(case))]
        return dict(case=case, batch=VolBatch(tiles, spot_sigma=case["spot"], outline_sigma=case["outline"]))
    shape = _shape(case)
    state = dict(case=case)
    if task in ("measure", "map"):
        state["labels"] = B200Array(_label_cells(shape, seed + 1).to(DTYPES[case["labels"]]))
    state["image"] = B200Array(_spots(shape, seed) if task == "voronoi" else _image(shape, case["dtype"], seed))
    return state


# ---- one pass ---------------------------------------------------------------
def _labels(tensor):
    """The label image's own memory as int32 (torch indexes no uint32)."""
    return tensor.view(torch.int32) if tensor.dtype == torch.uint32 else tensor


def run(state):
    case = state["case"]
    task = case["task"]
    if task == "tiles":
        return [_labels(t) for t in state["batch"].run()]
    image = state["image"]
    if task == "segment":
        return _labels(cle.voronoi_otsu_labeling(image, spot_sigma=case["spot"], outline_sigma=case["outline"]).tensor)
    if task == "measure":
        return cle.statistics_of_labelled_pixels(image, state["labels"])
    if task == "dense":
        return _labels(cle.gauss_otsu_labeling(image, outline_sigma=case["outline"]).tensor)
    if task == "blur":
        return cle.gaussian_blur(image, sigma_x=case["sx"], sigma_y=case["sy"], sigma_z=case["sz"]).tensor
    if task == "top_hat":
        return cle.top_hat_box(image, radius_x=case["rx"], radius_y=case["ry"], radius_z=case["rz"]).tensor
    if task == "voronoi":
        return _labels(cle.voronoi_labeling(image).tensor)
    return cle.label_mean_intensity_map(image, state["labels"]).tensor


def _taps(sigma):
    return int(sigma * 8.0) | 1 if sigma > 0 else 1


def work(case):
    task = case["task"]
    if task == "tiles":
        n, dims = sum(math.prod(s) for s in _tile_shapes(case)), 3
    else:
        n, dims = math.prod(_shape(case)), 3 if case["d"] else 2
    src = BYTES[case["dtype"]]
    if task in ("segment", "tiles"):
        sigmas = {case["spot"], case["outline"]}
        flops = sum(2 * dims * _taps(s) for s in sigmas) * n
        return {"bytes": (src + 4) * n, "flops": flops}
    if task == "dense":
        return {"bytes": (src + 4) * n, "flops": 2 * dims * _taps(case["outline"]) * n}
    if task == "blur":
        flops = 2 * n * sum(_taps(case[k]) for k in ("sx", "sy", "sz")[:dims])
        return {"bytes": (src + 4) * n, "flops": flops}
    if task == "measure":
        return {"bytes": (src + 4) * n, "flops": 0}
    if task == "map":
        return {"bytes": (src + 4 + 4) * n, "flops": 0}
    return {"bytes": (src + 4) * n, "flops": 0}     # top_hat, voronoi


# ---- the same in 64 bits ----------------------------------------------------
def _exact_blur(x, sigma, axis):
    n = _taps(sigma)
    if n == 1 and not sigma > 0:
        return x
    r = (n - 1) // 2
    w = [math.exp(-i * i / (2.0 * sigma * sigma)) for i in range(-r, r + 1)]
    total, size = sum(w), x.shape[axis]
    at = torch.arange(size, device=x.device)
    out = torch.zeros_like(x)
    for i in range(-r, r + 1):
        out.add_(x.index_select(axis, (at + i).clamp_(0, size - 1)), alpha=w[i + r] / total)
    return out


def _exact_box(x, r, axis, largest):
    """Largest (smallest) value within r of each place along an axis."""
    if r <= 0:
        return x
    size = x.shape[axis]
    at = torch.arange(size, device=x.device)
    out = x.clone()
    for i in range(-r, r + 1):
        y = x.index_select(axis, (at + i).clamp_(0, size - 1))
        out = torch.maximum(out, y) if largest else torch.minimum(out, y)
    return out


def _exact_statistics(image, labels):
    flat = labels.reshape(-1).to(torch.int64)
    at = flat.nonzero().view(-1)
    l = flat[at] - 1
    n = int(flat.max())
    v = image.reshape(-1).to(torch.float32)[at].double()
    shape = tuple(labels.shape) if labels.dim() == 3 else (1,) + tuple(labels.shape)
    pos = {"x": (at % shape[2]).double(), "y": (at // shape[2] % shape[1]).double(),
           "z": (at // (shape[1] * shape[2])).double()}

    def total(a):
        return torch.zeros(n, dtype=torch.float64, device=a.device).index_add_(0, l, a)

    def extreme(a, how):
        return torch.zeros(n, dtype=torch.float64, device=a.device).scatter_reduce_(0, l, a, how, include_self=False)

    area, s = total(torch.ones_like(v)), total(v)
    out = {"area": area, "sum_intensity": s, "mean_intensity": s / area, "min_intensity": extreme(v, "amin"),
           "max_intensity": extreme(v, "amax")}
    out["standard_deviation_intensity"] = (total((v - out["mean_intensity"][l]) ** 2) / area).sqrt()
    centroid, mass = torch.zeros_like(v), torch.zeros_like(v)
    for k, size in (("x", "width"), ("y", "height"), ("z", "depth")):
        p = pos[k]
        out["bbox_min_" + k], out["bbox_max_" + k] = extreme(p, "amin"), extreme(p, "amax")
        out["bbox_" + size] = out["bbox_max_" + k] - out["bbox_min_" + k] + 1
        out["sum_" + k], out["sum_intensity_times_" + k] = total(p), total(p * v)
        out["centroid_" + k], out["mass_center_" + k] = out["sum_" + k] / area, out["sum_intensity_times_" + k] / s
        centroid += (p - out["centroid_" + k][l]) ** 2
        mass += (p - out["mass_center_" + k][l]) ** 2
    for k, d in (("centroid", centroid.sqrt()), ("mass_center", mass.sqrt())):
        out["sum_distance_to_" + k], out["max_distance_to_" + k] = total(d), extreme(d, "amax")
        out["mean_distance_to_" + k] = out["sum_distance_to_" + k] / area
        out["mean_max_distance_to_" + k + "_ratio"] = out["max_distance_to_" + k] / out["mean_distance_to_" + k]
    out = {k: x.cpu().numpy() for k, x in out.items()}
    out["label"] = out["original_label"] = None      # whole numbers, compared as they are
    return out


def exact(case, seed):
    task = case["task"]
    if task not in ("measure", "blur", "top_hat", "map"):
        return None        # labels: whole numbers
    shape, seed = _shape(case), int(seed)
    image = _image(shape, case["dtype"], seed)
    if task == "blur":
        x = image.to(torch.float32).double()
        for k, axis in list(zip(("sx", "sy", "sz"), (-1, -2, -3)))[:len(shape)]:
            x = _exact_blur(x, case[k], axis)
        return x
    if task == "top_hat":
        x = f = image.to(torch.float32).double()
        for largest in (False, True):
            for k, axis in list(zip(("rx", "ry", "rz"), (-1, -2, -3)))[:len(shape)]:
                x = _exact_box(x, int(case[k]), axis, largest)
        return f - x
    labels = _label_cells(shape, seed + 1)
    if task == "measure":
        return _exact_statistics(image, labels)
    flat = labels.reshape(-1).to(torch.int64)
    n = int(flat.max()) + 1
    total = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(
        0, flat, image.reshape(-1).to(torch.float32).double())
    mean = total / torch.bincount(flat, minlength=n)
    mean[0] = 0
    return mean[flat].view(shape)
