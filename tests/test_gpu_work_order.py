"""GPU test of the order in which the blend takes the tiles: lists of every class of length, and more tiles than are handed out one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# 63,000 tiles of 8x8 pixels (several per visit of a warp, those of the long classes one by one) and 2,900
@pytest.mark.parametrize("width, height", [(2400, 1680), (504, 368)])
@pytest.mark.parametrize("mode", [0, 1])
def test_tiles_of_every_class_of_length(width, height, mode):
    import inpc_b200
    from inpc_b200.views import look_at_view
    g = torch.Generator().manual_seed(width + mode)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, height, float(width), float(width)).to(DEV)
    ty, tx = torch.meshgrid(torch.arange(4, height, 8, dtype=torch.float32), torch.arange(4, width, 8, dtype=torch.float32), indexing="ij")
    lengths = torch.ones(tx.numel(), dtype=torch.long)
    lengths[::3] = 0
    some = torch.randperm(tx.numel(), generator=g)
    for k, length in enumerate((63, 64, 65, 255, 256, 257, 600, 1023, 1024, 1025, 3000)):
        lengths[some[4 * k:4 * k + 4]] = length
    px, py = tx.reshape(-1).repeat_interleave(lengths), ty.reshape(-1).repeat_interleave(lengths)
    n = px.numel()
    px, py, z = px + torch.rand(n, generator=g) * 6 - 3, py + torch.rand(n, generator=g) * 6 - 3, torch.rand(n, generator=g)
    order = torch.randperm(n, generator=g)
    pos = torch.stack([(px - width / 2) / width * (3 - z), -(py - height / 2) / width * (3 - z), z], dim=1)[order].contiguous().to(DEV)
    feats = (torch.randn((n, 36), generator=g) * 0.5).to(torch.float16).to(DEV)
    opac = (torch.rand((n, 1), generator=g) * 0.05).to(DEV)
    gi, ga = torch.randn((4, height, width), generator=g).to(DEV), torch.randn((1, height, width), generator=g).to(DEV)
    out = []
    for tile in (8, 16):   # nothing depends on the tile size but the order of the sums
        f, o = feats.clone().requires_grad_(True), opac.clone().requires_grad_(True)
        image, alpha, weights = inpc_b200.INPCRasterizer(tile_size=tile)(view, mode, pos, f, o)
        torch.autograd.backward([image, alpha], [gi, ga])
        out.append((image.detach(), alpha.detach(), weights, o.grad, f.grad.float()))
    for a, b in zip(*out):
        # products of up to 3000 factors in another grouping: 3000 * 2^-24, times the size of the sums they stand in
        assert float((a - b).norm()) <= 1e-4 * float(b.norm())


# The blocks of a pass that stay for the whole of it are those that fit the chip (of gaussian forward passes three per multiprocessor at most), by the registers
# and shared memory of the kernel: of 2048 threads, 65536 registers (a
# warp takes them in units of 256) and 228 KB of shared memory (units of 128 bytes, 1 KB of every block for the system) per multiprocessor
def test_blend_passes_launch_the_blocks_that_are_resident(tmp_path):
    import json
    import inpc_b200
    from inpc_b200.views import look_at_view
    from torch.profiler import ProfilerActivity, profile
    n, side = 3000, 64
    g = torch.Generator().manual_seed(0)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), side, side, float(side), float(side)).to(DEV)
    pos, opac = (torch.rand((n, 3), generator=g) - 0.5).to(DEV), (torch.rand((n, 1), generator=g) * 0.3).to(DEV)
    rast = inpc_b200.INPCRasterizer()

    def passes():
        for mode in (0, 1):
            f, o = torch.zeros((n, 36), dtype=torch.float16, device=DEV).requires_grad_(True), opac.clone().requires_grad_(True)
            image, alpha, _ = rast(view, mode, pos, f, o)
            (image.sum() + alpha.sum()).backward()
            rast.render_preextracted(view, mode, pos, f.detach(), opac)
        for channels in (4, 8, 16, 32):
            f, o = torch.zeros((n, channels), device=DEV).requires_grad_(True), opac.clone().requires_grad_(True)
            image, alpha, _ = rast.forward_rows(view, pos, f, o)
            (image.sum() + alpha.sum()).backward()

    passes()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        passes()
        torch.cuda.synchronize()
    p.export_chrome_trace(str(tmp_path / "trace.json"))
    events = json.loads((tmp_path / "trace.json").read_text())["traceEvents"]
    seen = {e["name"].split("blend_", 1)[1].split("(")[0] + " " + str(e["args"].get("shared memory")): e["args"] for e in events
            if "blend" in e.get("name", "") and ("warp_forward" in e["name"] or "warp_backward" in e["name"]) and "grid" in e.get("args", {})}
    if not seen:
        pytest.skip("no activity records of kernels here")
    multiprocessors = torch.cuda.get_device_properties(0).multi_processor_count
    for name, a in seen.items():
        threads, registers, shared = a["block"][0], a["registers per thread"], a["shared memory"]
        fit = min(2048 // threads, 65536 // (-(-registers * 32 // 256) * 256 * threads // 32), 228 * 1024 // (-(-(shared + 1024) // 128) * 128))
        if "gaussian_warp_forward" in name:
            fit = min(fit, 3)
        assert a["grid"][0] == multiprocessors * fit, (name, a["grid"][0] / multiprocessors, fit)


# Which form a training step takes, on both sides of each line: images of 4096 tiles, 4160, 16384, 16640 and 33280, and the points per tile from which two warps take an item
@pytest.mark.parametrize("mode, channels, least, lines", [(0, None, 128, [(512, 512, True), (520, 512, None), (4096, 520, False)]), (0, 8, 32, [(512, 512, True), (520, 512, None), (4096, 520, False)]),
                                                          (1, None, 64, [(1024, 1024, True), (1040, 1024, None)])])
def test_where_two_warps_take_an_item(mode, channels, least, lines):
    import inpc_b200
    from inpc_b200.views import look_at_view
    from torch.profiler import ProfilerActivity, profile
    rast = inpc_b200.INPCRasterizer()

    def step(width, height, n):
        view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, height, float(width), float(width)).to(DEV)
        pos, opac = torch.full((n, 3), 9.0, device=DEV), torch.full((n, 1), 0.1, device=DEV).requires_grad_(True)      # (behind the camera: the rule asks how many there are)
        f = torch.zeros((n, channels), device=DEV) if channels else torch.zeros((n, 36), dtype=torch.float16, device=DEV)
        f.requires_grad_(True)
        image, alpha, _ = rast.forward_rows(view, pos, f, opac) if channels else rast(view, mode, pos, f, opac)
        (image.sum() + alpha.sum()).backward()

    step(64, 64, 10)
    for width, height, always in lines:
        tiles = width * height // 64
        for n in (least * tiles - 1, least * tiles):
            with profile(activities=[ProfilerActivity.CUDA]) as p:
                step(width, height, n)
                torch.cuda.synchronize()
            names = [e.key for e in p.key_averages()]
            if not any("inpc" in k for k in names):
                pytest.skip("no activity records of kernels here")
            paired = always if always is not None else n >= least * tiles
            forward = [k for k in names if "blend" in k and "forward" in k]
            assert sum("_pair_forward" in k for k in forward) == (2 if paired else 0), (width, height, n, forward)
            assert sum("_warp_forward" in k for k in forward) == (1 if paired else 3), (width, height, n, forward)
            if mode == 0 and not channels:
                assert any("blend_bilinear_pair_backward" in k for k in names) == paired


# Images are not cleared beforehand: tiles without instances are blanked at the end.  Into memory full of NaN; odd sizes; nothing, one point, all points culled, a few tiles with lists
# of one and of several segments among many empty ones
@pytest.mark.parametrize("width, height", [(8, 8), (101, 53), (1237, 40)])
@pytest.mark.parametrize("n", [0, 1, 40, 9000])
@pytest.mark.parametrize("mode", [0, 1])
def test_empty_tiles_are_blank_in_memory_that_is_not(width, height, n, mode):
    import inpc_b200
    from inpc_b200.views import look_at_view
    g = torch.Generator().manual_seed(n + width)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, height, float(width), float(width)).to(DEV)
    spot = torch.rand(n, generator=g) < 0.7                       # most points in one place, the others in a strip of the image
    px = torch.where(spot, width * 0.3 + torch.rand(n, generator=g) * 4, torch.rand(n, generator=g) * width * 0.4)
    py = torch.where(spot, height * 0.5 + torch.rand(n, generator=g) * 2, torch.rand(n, generator=g) * height)
    pos = torch.stack([(px - width / 2) / width * 3, -(py - height / 2) / width * 3, torch.zeros(n)], dim=1).contiguous().to(DEV)
    behind = pos + torch.tensor([0.0, 0.0, 9.0], device=DEV)
    feats, raw = ((torch.randn((n, k), generator=g) * 0.1 + 1.0).to(torch.float16).to(DEV) for k in (36, 37))
    opac, rows = torch.full((n, 1), 0.01, device=DEV), torch.ones((n, 8), device=DEV)
    rast = inpc_b200.INPCRasterizer()

    def calls(p):
        yield rast(view, mode, p, feats, opac)[:2]
        yield rast.render_preextracted(view, mode, p, feats, opac)
        yield rast.render(view, mode, p, raw, 1.0, 3.0)
        if mode == 0:
            yield rast.forward_rows(view, p, rows, opac)[:2]
            yield rast.render_multi(view, [(p, raw), (behind, raw), (p, raw)])

    def dirty():
        for k in (1, 4, 8, 3, 12):
            for _ in range(4):
                torch.full((k, height, width), float("nan"), device=DEV)

    for p in (pos, behind):
        torch.cuda.empty_cache()
        dirty()
        for out in calls(p):
            alpha = out[-1].reshape(-1, height, width)
            for t in out:
                assert bool(torch.isfinite(t).all())
                planes = t.reshape(alpha.shape[0], -1, height, width)
                assert bool((planes.transpose(0, 1)[:, alpha == 0.0] == 0.0).all())
            assert bool((alpha[:, :, int(width * 0.45) + 8:] == 0.0).all())
            if p is behind or n == 0:
                assert bool((alpha == 0.0).all())
            elif n > 30:
                assert bool((alpha[0] > 0.0).any())
            dirty()
