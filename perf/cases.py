"""The work that a user of this package has it do, as cases that can be timed: training steps (sampling, rasterization
forward and backward, octree statistics) from a few thousand samples to a batch of views, inference from a point cloud
and from multisampled sets, the export of a global cloud, and the loss and weight decay of a training iteration.

`listed` gives the cases, `draw` others of the same ranges; `prepare` makes what a program holds before the call, `run`
makes one pass through the public entry points, `work` counts the bytes and operations a pass cannot do without and
`tolerance` how far another correct implementation may be off.
"""
import math

import torch

from inpc_b200 import (INPCRasterizer, ProbabilityFieldSampler, add_normalized_weight_decay_grads, fused_cauchy_loss,
                       spherical_contraction)
from inpc_b200.batch import ViewShardedTrainer
from inpc_b200.compose import compose_background, render_multisampled
from inpc_b200.probability_field import prune, subdivide, update, update_from_samples
from inpc_b200.sampling import extract_global
from inpc_b200.views import look_at_view

BILINEAR, GAUSSIAN = 0, 1
DEVICE = "cuda"
PRUNE_THRESHOLD = 0.25      # of the mean leaf weight
SUBDIVIDE_THRESHOLD = 0.8


def listed():
    return [
        # one training step of a toy field: every launch and every line of Python counts
        dict(name="train_tiny", kind="train", points=1 << 14, leaves=4096, width=256, height=256, mode=BILINEAR, tile=8),
        # a step with a million samples of a smaller photograph, none of the sizes a multiple of anything
        dict(name="train_ragged", kind="train", points=1_000_003, leaves=100_003, width=801, height=533, mode=BILINEAR, tile=8),
        # the training step at the default sample count: 2^23 samples of a 2^18-leaf octree into 1237x822
        dict(name="train_full", kind="train", points=1 << 23, leaves=1 << 18, width=1237, height=822, mode=BILINEAR, tile=8),
        # the same step with gaussian splats, at half the samples
        dict(name="train_gaussian", kind="train", points=1 << 22, leaves=1 << 18, width=1237, height=822, mode=GAUSSIAN, tile=8),
        # a 4K training view of which nine tenths of the points crowd one corner of space: load imbalance, deep lists
        dict(name="train_skewed_4k", kind="skewed", points=1 << 24, width=3840, height=2160, mode=BILINEAR, tile=8),
        # wide feature rows: 16 fp32 channels blended as they are
        dict(name="train_rows16", kind="rows", points=1 << 23, leaves=1 << 18, width=1237, height=822, channels=16, tile=8),
        # one GPU's share of a 64-view batch on eight GPUs, pipelined over four streams
        dict(name="train_batch8", kind="batch", points=1 << 23, leaves=1 << 18, width=1237, height=822, views=8),
        # a frame of a viewer walking through a pre-extracted global cloud of the default size
        dict(name="render_cloud", kind="cloud", points=1 << 25, width=1920, height=1080, mode=BILINEAR, scales=False, tile=8),
        # a frame of a smaller cloud drawn as gaussian splats with a size per point
        dict(name="render_cloud_gaussian", kind="cloud", points=2_000_003, width=1297, height=840, mode=GAUSSIAN, scales=True, tile=8),
        # a high-quality frame: four sample sets drawn, rasterized and averaged over a background
        dict(name="render_multisampled", kind="multisample", points=1 << 23, leaves=1 << 18, width=1237, height=822, sets=4),
        # the end of training: prune, subdivide, and export of a global cloud over the training views
        dict(name="field_export", kind="field", points=1 << 25, leaves=1 << 18, views=16),
        # what a training iteration does outside the renderer: compose over the background, loss, gradients, and weight
        # decay on the ten-level hash grid
        dict(name="loss_and_decay", kind="loss", params=210_917_376, width=1237, height=822),
    ]


def _log_int(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, v + (rng.random() < 0.5)))


def _image(rng, lo, hi):
    w = _log_int(rng, lo, hi)
    return w, max(lo // 2, int(w * rng.uniform(0.55, 0.8)))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "skewed", "rows", "batch", "cloud", "cloud", "multisample", "field", "loss"])
    w, h = _image(rng, 200, 1400)
    tile = 16 if rng.random() < 0.15 else 8
    leaves = _log_int(rng, 4096, 1 << 18)
    if kind == "train":
        gaussian = rng.random() < 0.3
        return dict(kind=kind, points=_log_int(rng, 1 << 13, 1 << (22 if gaussian else 23)), leaves=leaves, width=w, height=h,
                    mode=GAUSSIAN if gaussian else BILINEAR, tile=tile)
    if kind == "skewed":
        w, h = _image(rng, 640, 3840)
        h = min(h, 2160)
        return dict(kind=kind, points=_log_int(rng, 1 << 18, 1 << 24), width=w, height=h, mode=BILINEAR, tile=tile)
    if kind == "rows":
        return dict(kind=kind, points=_log_int(rng, 1 << 14, 1 << 23), leaves=leaves, width=w, height=h,
                    channels=rng.choice([4, 8, 16, 16, 32]), tile=tile)
    if kind == "batch":
        return dict(kind=kind, points=_log_int(rng, 1 << 16, 1 << 22), leaves=leaves, width=w, height=h, views=rng.randint(4, 16))
    if kind == "cloud":
        w, h = _image(rng, 320, 1920)
        h = min(h, 1080)
        gaussian = rng.random() < 0.4
        return dict(kind=kind, points=_log_int(rng, 1 << 15, 1 << (22 if gaussian else 25)), width=w, height=h,
                    mode=GAUSSIAN if gaussian else BILINEAR, scales=gaussian and rng.random() < 0.7, tile=tile)
    if kind == "multisample":
        sets = rng.randint(2, 8)
        return dict(kind=kind, points=_log_int(rng, 1 << 15, (1 << 25) // sets), leaves=leaves, width=w, height=h, sets=sets)
    if kind == "field":
        return dict(kind=kind, points=_log_int(rng, 1 << 18, 1 << 25), leaves=leaves, views=rng.randint(1, 64))
    return dict(kind="loss", params=_log_int(rng, 1 << 18, 210_917_376), width=w, height=h)


# ---- inputs ---------------------------------------------------------------------------------------------------------

def _generator(seed, salt=0):
    return torch.Generator(device=DEVICE).manual_seed(seed * 64 + salt)


def _normal(shape, g, std=1.0, mean=0.0):
    return torch.randn(shape, generator=g, device=DEVICE).mul_(std).add_(mean)


class _Octree:
    """A carved adaptive octree in [-1,1]^3: random cells of `base` cells a side, half of the cells of every level split
    again down to `base * 2^depth`, trimmed to `leaves`; weights softmax(N(0,2)).  `centers`, `levels`, `weights` and
    `initial_size` are what the sampler takes."""

    def __init__(self, leaves, seed, relative=False):
        g = _generator(seed, 1)
        base_level, depth = (6, 4) if leaves > 1 << 15 else (4, 3)
        per_cell = sum(0.5 * 4 ** k for k in range(depth)) + 4 ** depth
        side = 1 << base_level
        start = torch.randperm(side ** 3, generator=g, device=DEVICE)[: min(side ** 3, int(leaves / per_cell * 1.02) + 3)]
        cells = torch.stack([start // (side * side), (start // side) % side, start % side], dim=1)
        corner = torch.tensor([[a, b, c] for a in (0, 1) for b in (0, 1) for c in (0, 1)], device=DEVICE)
        done, done_level = [], []
        for k in range(depth):
            order = torch.randperm(cells.shape[0], generator=g, device=DEVICE)
            half = (cells.shape[0] + 1) // 2
            done.append(cells[order[half:]])
            done_level.append(torch.full((cells.shape[0] - half,), k, dtype=torch.int32, device=DEVICE))
            parents = cells[order[:half].sort().values]
            cells = (parents[:, None, :] * 2 + corner[None]).reshape(-1, 3)
        done.append(cells)
        done_level.append(torch.full((cells.shape[0],), depth, dtype=torch.int32, device=DEVICE))
        cells, level = torch.cat(done), torch.cat(done_level)
        keep = torch.randperm(cells.shape[0], generator=g, device=DEVICE)[:leaves].sort().values
        cells, level = cells[keep], level[keep]
        edge = 2.0 / side / torch.exp2(level.float())
        self.centers = ((cells.float() + 0.5) * edge[:, None] - 1.0).contiguous()
        self.levels = (level if relative else level + base_level).contiguous()
        self.initial_size = 2.0 / side if relative else 2.0
        self.weights = torch.softmax(_normal((self.centers.shape[0],), g, 2.0), dim=0)


def _orbit(azimuth, elevation, width, height, focal, radius=3.0):
    eye = (radius * math.cos(elevation) * math.sin(azimuth), radius * math.sin(elevation),
           radius * math.cos(elevation) * math.cos(azimuth))
    return look_at_view(eye, (0.0, 0.0, 0.0), width, height, focal, focal, device=DEVICE)


def _views(count, seed, width, height):
    g = torch.Generator().manual_seed(seed * 64 + 2)
    az, el = torch.rand(count, generator=g) * (2 * math.pi), (torch.rand(count, generator=g) - 0.5) * (math.pi / 3)
    return [_orbit(float(a), float(e), width, height, 960.0 * width / 1237) for a, e in zip(az, el)]


def _upstream(channels, height, width, g):
    """Upstream gradients of an image and its alpha, as the network behind the renderer hands them back."""
    return _normal((channels, height, width), g, 1e-3), _normal((1, height, width), g, 1e-3)


def _chunked_half(n, width, g, std, mean=0.0):
    out = torch.empty((n, width), dtype=torch.float16, device=DEVICE)
    for a in range(0, n, 1 << 22):
        out[a:a + (1 << 22)] = _normal((min(n, a + (1 << 22)) - a, width), g, std, mean)
    return out


def prepare(case, seed):
    kind = case["kind"]
    g = _generator(seed, 3)
    s = dict(case)
    if kind in ("train", "rows", "batch", "multisample", "field"):
        s["tree"] = tree = _Octree(case["leaves"], seed, relative=kind == "field")
    if "tile" in case:
        s["rasterizer"] = INPCRasterizer(tile_size=case["tile"])
    if kind in ("train", "skewed", "rows", "batch"):
        n, w, h = case["points"], case["width"], case["height"]
        rows = kind == "rows"
        s["features"] = _normal((n, case["channels"]), g, 0.5) if rows else _chunked_half(n, 36, g, 0.5)
        s["opacities"] = torch.sigmoid(_normal((n, 1), g, 1.0, 2.0 if kind == "skewed" else 0.0))
        s["grad_image"], s["grad_alpha"] = _upstream(case.get("channels", 4), h, w, g)
        s["background"] = torch.rand((case.get("channels", 4), h, w), generator=g, device=DEVICE)
    if kind in ("train", "rows", "batch"):
        s["sampler"] = ProbabilityFieldSampler(seed)
        # the octree's occupancy as the optimiser keeps it; the weights that are drawn from stay as they are, so that
        # every pass is the same amount of work
        s["occupancy"], s["scores"] = tree.weights.clone(), torch.zeros_like(tree.weights)
    if kind in ("train", "rows", "multisample"):
        s["view"] = _views(1, seed, case["width"], case["height"])[0]
    if kind == "skewed":
        n = case["points"]
        hot = int(n * 0.9)
        p = torch.cat([_normal((hot, 3), g, 0.02) + torch.tensor([0.0, 0.0, 2.0], device=DEVICE),
                       torch.rand((n - hot, 3), generator=g, device=DEVICE) * 2 - 1])
        s["positions"] = p[torch.randperm(n, generator=g, device=DEVICE)].contiguous()
        s["view"] = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), case["width"], case["height"], 2800.0 * case["width"] / 3840,
                                 2800.0 * case["width"] / 3840, device=DEVICE)
    if kind == "batch":
        s["views"] = _views(case["views"], seed, case["width"], case["height"])
        s["trainer"] = ViewShardedTrainer(tree, s["features"], s["opacities"], case["points"], seed)
    if kind == "cloud":
        n = case["points"]
        mu = torch.rand((64, 3), generator=g, device=DEVICE) * 2 - 1
        s["positions"] = (mu[torch.randint(0, 64, (n,), generator=g, device=DEVICE)] + _normal((n, 3), g, 0.1)).contiguous()
        s["features"] = _chunked_half(n, 36, g, 0.3, 0.5)
        s["opacities"] = torch.rand((n, 1), generator=g, device=DEVICE) * 0.9 + 0.05
        focal = 1400.0 * case["width"] / 1920
        # around one pixel at the scene's distance
        s["splat_scales"] = torch.exp(_normal((n, 1), g, 0.5)) * (3.0 / focal) if case["scales"] else None
        s["view"] = look_at_view((0.0, 0.5, 3.0), (0.0, 0.0, 0.0), case["width"], case["height"], focal, focal, device=DEVICE)
    if kind == "multisample":
        s["sampler"] = ProbabilityFieldSampler(seed)
        s["rasterizer"] = INPCRasterizer()
        t = tree
        n = ProbabilityFieldSampler(seed).generate_expected_samples(t.centers, t.levels, t.weights, s["view"], case["points"], 1,
                                                                    t.initial_size).shape[0]
        # what the appearance network returns for every set: log-density and SH coefficients
        s["features_raw"] = [_chunked_half(n, 37, g, 0.5) for _ in range(case["sets"])]
        s["background"] = torch.rand((4, case["height"], case["width"]), generator=g, device=DEVICE)
    if kind == "field":
        s["views"] = _views(case["views"], seed, 1237, 822)
        s["sampler"] = ProbabilityFieldSampler(seed)
        # the quantiles of the weights and scores, dealt out at random: how many leaves pass a threshold is the same for every
        # seed, which ones is not
        leaves = tree.weights.shape[0]
        quantile = (torch.arange(leaves, device=DEVICE, dtype=torch.float32) + 0.5) / leaves
        deal = torch.randperm(leaves, generator=g, device=DEVICE)
        tree.weights = torch.softmax(torch.erfinv(2 * quantile - 1) * (2.0 * math.sqrt(2.0)), dim=0)[deal].contiguous()
        s["scores"] = torch.frac(torch.arange(leaves, device=DEVICE, dtype=torch.float64) * 0.6180339887498949).float()[deal].contiguous()
    if kind == "loss":
        h, w = case["height"], case["width"]
        s["image"], s["background"], s["target"] = (torch.rand((3, h, w), generator=g, device=DEVICE) for _ in range(3))
        s["alpha"] = torch.rand((1, h, w), generator=g, device=DEVICE)
        s["grid"] = torch.nn.Parameter(_normal((case["params"],), g, 0.1))
        s["grid"].grad = _normal((case["params"],), g, 1e-3)
    return s


# ---- one pass -------------------------------------------------------------------------------------------------------

def _sample(s):
    t = s["tree"]
    return s["sampler"].generate_training_samples(t.centers, t.levels, t.weights, s["view"], s["points"], t.initial_size)


def _backward(s, image, alpha):
    composed = compose_background(image, alpha, s["background"])
    torch.autograd.backward([composed, alpha], [s["grad_image"], s["grad_alpha"]])
    return composed


def run(s):
    kind = s["kind"]
    if kind in ("train", "rows", "skewed"):
        features, opacities = s["features"].detach().requires_grad_(True), s["opacities"].detach().requires_grad_(True)
        out = {}
        if kind == "skewed":
            positions = s["positions"]
        else:
            positions, indices = _sample(s)
            out.update(positions=positions, indices=indices, contracted=spherical_contraction(positions))
        if kind == "rows":
            image, alpha, weights = s["rasterizer"].forward_rows(s["view"], positions, features, opacities)
        else:
            image, alpha, weights = s["rasterizer"](s["view"], s["mode"], positions, features, opacities)
        composed = _backward(s, image, alpha)
        if kind != "skewed":
            update_from_samples(s["occupancy"], s["scores"], indices, weights)
            out.update(occupancy=s["occupancy"], scores=s["scores"])
        out.update(image=composed, alpha=alpha, weights=weights, grad_features=features.grad, grad_opacities=opacities.grad)
        return out
    if kind == "batch":
        trainer = s["trainer"]
        image, alpha, weights, grad_features, grad_opacities = trainer.run_batch(s["views"], (s["grad_image"], s["grad_alpha"]))
        update(s["occupancy"], s["scores"], trainer.buffers.leaf)
        return dict(image=image, alpha=alpha, weights=weights, grad_features=grad_features, grad_opacities=grad_opacities,
                    appearance=trainer.buffers.appearance, occupancy=s["occupancy"], scores=s["scores"])
    if kind == "cloud":
        return s["rasterizer"].render_preextracted(s["view"], s["mode"], s["positions"], s["features"], s["opacities"], s["splat_scales"])
    if kind == "multisample":
        t, k = s["tree"], s["sets"]
        positions = s["sampler"].generate_expected_samples(t.centers, t.levels, t.weights, s["view"], s["points"], k, t.initial_size)
        sets = list(zip(positions.chunk(k), s["features_raw"]))
        return render_multisampled(s["rasterizer"], s["view"], BILINEAR, sets, s["background"], n_streams=2, batched=True)
    if kind == "field":
        t = s["tree"]
        centers, levels, weights, scores = prune(t.centers, t.levels, t.weights, s["scores"], PRUNE_THRESHOLD / t.weights.shape[0])
        centers, levels, weights, scores = subdivide(centers, levels, weights, scores, SUBDIVIDE_THRESHOLD, t.initial_size)
        cloud = extract_global(s["sampler"], centers, levels, weights, s["views"], s["points"], t.initial_size)
        return centers, levels, weights, scores, cloud
    image, alpha = s["image"].detach().requires_grad_(True), s["alpha"].detach().requires_grad_(True)
    loss = fused_cauchy_loss(compose_background(image, alpha, s["background"]), s["target"])
    loss.backward()
    add_normalized_weight_decay_grads(s["grid"])
    return dict(loss=loss, grad_image=image.grad, grad_alpha=alpha.grad, grad_grid=s["grid"].grad)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------

# Operations per point: three affine rows and two divisions (25), SH basis and four channels of nine coefficients (30 + 72),
# and per bilinear splat four fragments of weight, alpha, transmittance and 2 C operations.  The backward pass does about
# twice the forward's.
def _point_flops(channels, backward):
    forward = 25 + 102 + 4 * (12 + 2 * channels)
    return 3 * forward if backward else forward


def work(case):
    kind = case["kind"]
    n, leaves = case.get("points", 0), case.get("leaves", 0)
    px = case.get("width", 0) * case.get("height", 0)
    c = case.get("channels", 4)
    row = 4 * c if kind == "rows" else 72
    # features and opacity in, their gradients and the blending weight out; image, alpha and their gradients
    train = n * (row + 4 + row + 4 + 4) + px * 4 * (2 * c + 2)
    if kind in ("train", "rows"):
        # the octree in and its occupancy in and out; positions (also contracted) and indices out; background in, composed image out
        return {"bytes": train + leaves * (20 + 16) + n * (12 + 12 + 8) + px * 4 * (2 * c), "flops": n * (_point_flops(c, True) + 60)}
    if kind == "skewed":
        return {"bytes": train + n * 12 + px * 4 * (2 * c), "flops": n * _point_flops(c, True)}
    if kind == "batch":
        # features, opacities and upstream gradients are the same for all views: read once; the gradients of every view exist
        return {"bytes": n * (72 + 4) + case["views"] * (n * (72 + 4 + 4 + 12 + 8) + px * 20) + px * 20 + leaves * (20 + 16) + 4 * (1 << 22),
                "flops": case["views"] * n * (_point_flops(4, True) + 40)}
    if kind == "cloud":
        return {"bytes": n * (12 + 72 + 4 + (4 if case["scales"] else 0)) + px * 24, "flops": n * _point_flops(4, False)}
    if kind == "multisample":
        return {"bytes": case["sets"] * n * (12 + 74) + leaves * 20 + px * (16 + 28), "flops": case["sets"] * n * (_point_flops(4, False) + 40)}
    if kind == "field":
        # the octree in, two fifths of it kept, a fifth of those split in eight: nine tenths as many leaves out; the cloud out
        return {"bytes": int(leaves * 24 * 2.3) + n * 12, "flops": n * 100 + case["views"] * leaves * 40}
    return {"bytes": case["params"] * 12 + px * 4 * (3 * 3 + 1 + 3 + 1), "flops": case["params"] * 2 + px * 60}


def tolerance(case):
    kind = case["kind"]
    if kind == "field":
        return "exact"      # integers, and positions whose roundings are all prescribed
    if kind == "loss":
        return {"rel": 1e-5}
    if kind in ("train", "skewed", "batch"):
        # 32-bit sums taken in another order move a feature gradient across a rounding boundary of its half now and then; the
        # smallest of them lie below the normal range of a half, where that one step is up to a hundredth of the root mean square
        return {"rel": 1e-4, "max": 0.02}
    # 32-bit sums; single values where a pixel's transmittance cancels (opacity gradients) or falls below its stop are less exact
    return {"rel": 1e-5, "max": 1e-3}
