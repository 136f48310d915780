"""The work a user has this framework do, as cases that can be timed and compared.

``train``      one optimizer step of the 3-D U-Net through :class:`TrainEngine` (forward, fused loss, backward, clip,
               Adam), the call the trainer and ``bench.py`` make once per batch
``validate``   one validation batch (``TrainEngine.eval_step``), as the evaluation pass runs it after every epoch
``predict``    the logits of a volume under bf16 autocast, as a user of a trained model takes them
``instances``  the point clouds of fractal instances (``scaffold generate_fractals``)
``volume``     one labelled volume rendered from point clouds (the dataset generation of ``scaffold benchmark``)

Volumes are sparse, as the dataset's are: a background of zeros and a few fractals of one colour each. The training
steps take no class weights, as ``bench.py``: with weights of about a hundred on a handful of voxels the gradients of a
network at its random start are sums of cancelling terms that bf16 does not determine to a few percent.
"""
from __future__ import annotations

import numpy as np
import torch

from scaffold_b200.data import category_search, ifs, instances, volumes
from scaffold_b200.models.unet import UNet
from scaffold_b200.ops.optim import FusedClipAdam
from scaffold_b200.train.engine import TrainEngine

POINTS_PER_VOXEL = 256  # a fractal instance has one point per 256 voxels of the volume (the configuration's rule)
FRACTALS_PER_VOLUME = 3
LEARNING_RATE = 1e-4  # the floor of the default schedule, where a long run spends most of its steps


def _net(kind, name, dims, layers, width, batch, classes, weights=False, recompute=False):
    return {"name": name, "kind": kind, "d": dims[0], "h": dims[1], "w": dims[2], "layers": layers, "width": width,
            "batch": batch, "classes": classes, "class_weights": weights, "recompute": recompute}


def listed():
    cube = lambda n: (n, n, n)  # noqa: E731
    return [
        # the smallest problem of the tests and the smoke run: scale 5, where launches and the host path count
        _net("train", "train 32 w64 b1", cube(32), 2, 64, 1, 6),
        # scale 6 with the default configuration's batch
        _net("train", "train 64 w64 b1", cube(64), 3, 64, 1, 6),
        # the default configuration: scale 7, five categories, batch 1
        _net("train", "train 128 w64 b1", cube(128), 4, 64, 1, 6),
        # the headline benchmark: scale 7, eight categories, batch 2
        _net("train", "train 128 w64 b2", cube(128), 4, 64, 2, 9),
        # scale 7 at base width 32, the narrow network that the time-to-Dice runs use
        _net("train", "train 128 w32 b2", cube(128), 4, 32, 2, 9),
        # scale 8 on one GPU: the largest problem that one sample per GPU gives
        _net("train", "train 256 w64 b1", cube(256), 5, 64, 1, 6),
        # a sub-volume whose extents are no powers of two (odd at two of the levels, so the decoder pads)
        _net("train", "train 44x60x76 w64 b2", (44, 60, 76), 3, 64, 2, 9),
        # the activation_checkpointing option, which runs every block's forward pass twice
        _net("train", "train 128 w64 b1 recompute", cube(128), 4, 64, 1, 6, recompute=True),
        # the validation pass of the headline configuration, with the trainer's class weights
        _net("validate", "validate 128 w64 b2", cube(128), 4, 64, 2, 9, weights=True),
        # a trained model applied to a volume of the user's own size
        _net("predict", "predict 100x84x116 w32 b1", (100, 84, 116), 4, 32, 1, 6),
        # all instances of the default configuration: five categories of 145 at scale 7
        {"name": "instances 725 x 8192", "kind": "instances", "orbits": 725, "points": 8192},
        # one volume of the default configuration
        {"name": "volume 128", "kind": "volume", "grid": 128, "clouds": FRACTALS_PER_VOLUME},
    ]


def draw(rng):
    kind = rng.choices(("train", "validate", "predict", "instances", "volume"), (12, 2, 3, 1, 1))[0]
    if kind == "instances":
        return {"kind": kind, "orbits": round(145 * 2 ** rng.uniform(0, 3.3)), "points": round(2 ** rng.uniform(9, 14))}
    if kind == "volume":
        return {"kind": kind, "grid": rng.choice((32, 48, 64, 96, 100, 128, 160, 192, 256)), "clouds": rng.randint(1, 5)}
    width = rng.choice((16, 32, 32, 64, 64, 64))
    voxels = 2 ** rng.uniform(15, 22)  # of the whole batch: 32 cubed to 2 x 128 cubed
    batch = rng.choice((1, 1, 2, 3, 4))
    edge = max(32.0, (voxels / batch) ** (1 / 3))
    if rng.random() < 0.4:  # cubes of a power of two, the datasets' own form
        dims = [2 ** round(np.log2(edge))] * 3
    else:
        dims = [max(24, round(edge * rng.uniform(0.7, 1.4))) for _ in range(3)]
    layers = rng.randint(2, 4 if min(dims) >= 64 else 3 if min(dims) >= 32 else 2)
    while batch > 1 and batch * dims[0] * dims[1] * dims[2] > 2 ** 22:
        batch -= 1
    case = _net(kind, "", dims, layers, width, batch, rng.randint(2, 17),
                kind == "validate" and rng.random() < 0.7, kind == "train" and rng.random() < 0.15)
    del case["name"]
    return case


# -- inputs ------------------------------------------------------------------------------------------------------------
def _fractal_batch(case, gen, dev):
    """(images fp32 [B, 3, D, H, W], masks int16 [B, D, H, W]): a few chaos-game clouds per volume."""
    b, dims = case["batch"], (case["d"], case["h"], case["w"])
    images = torch.zeros((b, 3, *dims), device=dev)
    masks = torch.zeros((b, *dims), dtype=torch.int16, device=dev)
    size = torch.tensor(dims, device=dev, dtype=torch.float32)
    n = max(64, dims[0] * dims[1] * dims[2] // POINTS_PER_VOXEL)
    for s in range(b):
        labels = torch.randint(1, case["classes"], (FRACTALS_PER_VOLUME,), generator=gen, device=dev)
        for label in labels:
            m = torch.rand((2, 3, 3), generator=gen, device=dev) * 1.1 - 0.55
            t = torch.rand((2, 3), generator=gen, device=dev) * 2 - 1
            p = torch.rand((n, 3), generator=gen, device=dev)
            for _ in range(14):
                pick = torch.rand(n, generator=gen, device=dev) < 0.5
                p = torch.where(pick[:, None], p @ m[0].T + t[0], p @ m[1].T + t[1])
            lo, hi = p.amin(0), p.amax(0)
            at = ((p - lo) / (hi - lo).clamp_min(1e-6) * (size - 1)).long()
            images[s][:, at[:, 0], at[:, 1], at[:, 2]] = torch.rand((3, 1), generator=gen, device=dev)
            masks[s][at[:, 0], at[:, 1], at[:, 2]] = label.to(torch.int16)
    return images, masks


def _class_weights(masks, classes):
    """total / background for class 0, total / foreground for the others: the trainer's rule."""
    total = masks.numel()
    fg = (masks > 0).sum().clamp(1, total - 1).float()
    w = torch.full((classes,), 0.0, device=masks.device)
    w[0], w[1:] = total / (total - fg), total / fg
    return w


def _contractive_maps(rng, count):
    p = rng.uniform(-1.0, 1.0, (count, 2, 13))
    a = p[:, :, :9].reshape(count, 2, 3, 3)
    a /= np.maximum(1.0, 1.3 * np.linalg.norm(a, 2, axis=(2, 3)))[:, :, None, None]
    det = np.abs(np.linalg.det(a)) + 1e-9
    p[:, :, :9], p[:, :, 12] = a.reshape(count, 2, 9), det / det.sum(1, keepdims=True)
    return p


def prepare(case, seed):
    if case["kind"] == "instances":
        rng = np.random.default_rng(seed)
        table = instances.instance_weights()
        categories = -(-case["orbits"] // len(table))
        params = np.repeat(_contractive_maps(rng, categories), len(table), 0)[:case["orbits"]]
        params[:, :, :12] *= np.tile(table, (categories, 1))[:case["orbits"], None]
        seeds = np.array([category_search.orbit_seed(seed, 0, i) for i in range(case["orbits"])], dtype=np.uint64)
        return {"case": case, "params": params, "seeds": seeds}
    if case["kind"] == "volume":
        rng = np.random.default_rng(seed)
        n, k = max(64, case["grid"] ** 3 // POINTS_PER_VOXEL), case["clouds"]
        clouds, _ = ifs.orbit_points(_contractive_maps(rng, k), rng.integers(1, 2 ** 62, k).astype(np.uint64), n)
        return {"case": case, "clouds": list(clouds), "cats": [int(c) for c in rng.integers(0, 5, k)],
                "colors": rng.random((5, 3))}
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(seed)
    images, masks = _fractal_batch(case, gen, dev)
    torch.manual_seed(seed)
    with dev:
        model = UNet(3, case["classes"], layers=case["layers"], base_width=case["width"])
    state = {"case": case, "images": images, "masks": masks, "model": model}
    if case["kind"] == "predict":
        model.eval()
        return state
    if case["recompute"]:
        model.use_checkpointing()
    weights = _class_weights(masks, case["classes"]) if case["class_weights"] else None
    optimizer = FusedClipAdam(model.parameters(), lr=LEARNING_RATE, max_norm=1.0)
    state["engine"] = TrainEngine(model, optimizer, case["classes"], dev, class_weights=weights)
    model.train(case["kind"] == "train")
    return state


# -- one pass ----------------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        engine = state["engine"]
        loss = engine.step(state["images"], state["masks"])
        return {"loss": loss, "weights": engine.flat.data, "grads": engine.flat.grad}
    if kind == "validate":
        loss, dice = state["engine"].eval_step(state["images"], state["masks"])
        return {"loss": loss, "dice": dice}
    if kind == "predict":
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return state["model"](state["images"])
    if kind == "instances":
        return ifs.orbit_points(state["params"], state["seeds"], case["points"], device="cuda")
    return volumes.render_volume_shard(state["clouds"], state["cats"], state["colors"], case["grid"], [1, 1, 1],
                                       [2, 3, 4], 0, "cuda")


# -- what a pass cannot do without -------------------------------------------------------------------------------------
def _convolutions(case):
    """(voxels of the output, multiply-adds per voxel, output channels, parameters) of every convolution."""
    dims = [[case["d"], case["h"], case["w"]]]
    for _ in range(case["layers"]):
        dims.append([v // 2 for v in dims[-1]])
    vox = [case["batch"] * d * h * w for d, h, w in dims]
    width, rows = case["width"], []
    for level in range(case["layers"] + 1):
        c = width << level
        cin = 3 if level == 0 else c // 2
        rows += [(vox[level], 27 * cin * c, c, 27 * cin * c), (vox[level], 27 * c * c, c, 27 * c * c)]
    for level in reversed(range(case["layers"])):
        c = width << level
        rows += [(8 * vox[level + 1], 2 * c * c, c, 16 * c * c), (vox[level], 27 * 2 * c * c, c, 54 * c * c),
                 (vox[level], 27 * c * c, c, 27 * c * c)]
    rows.append((vox[0], width * case["classes"], case["classes"], width * case["classes"]))
    return vox[0], rows


def work(case):
    """Bytes and operations of one pass. A network pass reads its volume and weights; a training step also writes and
    reads back every feature map once (bf16, for the backward pass) and reads and writes the optimizer's state."""
    if case["kind"] == "instances":
        n = case["orbits"] * case["points"]
        return {"bytes": 12 * n, "flops": 18 * n}
    if case["kind"] == "volume":
        vox = case["grid"] ** 3
        n = case["clouds"] * max(64, vox // POINTS_PER_VOXEL)
        return {"bytes": 14 * vox + 12 * n, "flops": 21 * n}
    vox, rows = _convolutions(case)
    fwd = sum(2 * v * macs for v, macs, _, _ in rows)
    params = sum(p for *_, p in rows)
    if case["kind"] == "predict":
        return {"bytes": 12 * vox + 4 * params + 2 * vox * case["classes"], "flops": fwd}
    if case["kind"] == "validate":
        return {"bytes": 14 * vox + 4 * params, "flops": fwd}
    first = 2 * rows[0][0] * rows[0][1]  # the first convolution needs no gradient of its input
    maps = sum(2 * v * c for v, _, c, _ in rows)
    flops = 3 * fwd - first + (fwd if case["recompute"] else 0)  # checkpointing is a second forward pass
    return {"bytes": 14 * vox + 2 * maps + 28 * params, "flops": flops}


def tolerance(case):
    """bf16 tensors with fp32 sums: the training step's gradients move by up to 0.3 % (2-norm) when the same step adds its
    sums in another order (two consecutive steps, the statistics passes separate and the wide layers on the single-CTA
    kernels), and lie up to 0.6 % from fp32 throughout; the logits move by 0.4 % and lie 0.7 % from fp32. A few single
    gradients that are sums of cancelling terms move by over half of the gradients' root mean square. The generators
    work in fp64 with a fixed order of operations, so their results are the same to the last bit."""
    if case["kind"] in ("instances", "volume"):
        return "exact"
    if case["kind"] == "train":
        return {"rel": 0.012, "max": 0.9}
    return {"rel": 0.02, "max": 0.6}
