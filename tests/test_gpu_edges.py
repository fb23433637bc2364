"""GPU tests at the sizes where a kernel's tiling can go wrong: tile edges, remainders, the smallest and the largest of a
dispatch range.  Integer results are compared exactly, the rest against the oracle with the tolerance stated."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# tiles of 2048 pairs up to 2^18 pairs, of 8192 above
@pytest.mark.parametrize("n", [2047, 2048, 2049, (1 << 18) - 1, 1 << 18, (1 << 18) + 1, 8192 * 37 + 1])
@pytest.mark.parametrize("end_bit", [9, 14, 27, 30])
def test_sort_at_the_edges_of_its_tiles(n, end_bit):
    from inpc_b200 import _cabi
    g = torch.Generator(device=DEV).manual_seed(n + end_bit)
    keys64 = torch.randint(0, 1 << 32, (n,), generator=g, device=DEV, dtype=torch.int64)
    k, v = keys64.to(torch.int32), torch.arange(n, device=DEV, dtype=torch.int32)
    ka, va = torch.empty_like(k), torch.empty_like(v)
    ws = torch.full((int(_cabi.lib().inpc_sort_workspace_bytes(n)),), 0xA5, dtype=torch.uint8, device=DEV)
    alt = C.c_int(0)
    _cabi.check(_cabi.lib().inpc_sort_pairs(k.data_ptr(), ka.data_ptr(), v.data_ptr(), va.data_ptr(), n, end_bit, ws.data_ptr(), C.byref(alt),
                                           torch.cuda.current_stream().cuda_stream))
    order = torch.sort(keys64 & ((1 << end_bit) - 1), stable=True).indices
    assert torch.equal((va if alt.value else v).to(torch.int64), order)
    assert torch.equal((ka if alt.value else k).to(torch.int64) & 0xFFFFFFFF, keys64[order])


# a block places 2048 consecutive samples; it keeps the offsets of at most 2048 leaves in shared memory
@pytest.mark.parametrize("total,gap,largest", [(1, 0, 1), (2047, 0, 39), (2048, 0, 39), (2048, 1, 39), (2049, 3000, 39), (6145, 2049, 39),
                                               (20_000, 2047, 39), (4096, 0, 2048), (300_001, 5, 300_000)])
def test_halton_samples_over_runs_of_empty_leaves(total, gap, largest):
    from inpc_b200.sampling import halton_samples
    g = torch.Generator().manual_seed(total)
    filled = torch.randint(1, largest + 1, (total,), generator=g)
    filled[0] = largest                                    # up to 300,000 samples in one leaf: many digits behind the tabulated ones
    filled = filled[:int((filled.cumsum(0) < total).sum()) + 1]
    filled[-1] -= int(filled.sum()) - total                # the last leaf takes what is left, at least one
    assert int(filled.sum()) == total and int(filled.min()) >= 1
    counts = torch.zeros(len(filled) * 2 + gap * 3, dtype=torch.int32)
    at = torch.arange(len(filled)) * 2
    at[len(filled) // 2:] += gap
    at[len(filled) * 3 // 4:] += gap
    counts[at] = filled.to(torch.int32)
    n = counts.numel()
    centers = torch.rand((n, 3), generator=g) * 2 - 1
    levels = torch.randint(0, 11, (n,), generator=g, dtype=torch.int32)
    out = halton_samples(counts.to(DEV), centers.to(DEV), levels.to(DEV), 2.0)
    assert out.shape == (total, 3)
    np.testing.assert_array_equal(out.cpu().numpy(), O.halton_samples(counts.numpy(), centers.numpy(), levels.numpy(), 2.0))


def _one_tile_scene(n, seed, width=24, height=16):
    """n faint points in front of the 24x16 pixels in the upper left corner of an image, three quarters of them over one 8x8 tile."""
    from inpc_b200.views import look_at_view
    g = torch.Generator().manual_seed(seed)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, height, 24.0, 24.0, center_x=12.0, center_y=8.0)
    z = torch.rand(n, generator=g) * 2 - 1
    px = torch.where(torch.rand(n, generator=g) < 0.75, 8 + torch.rand(n, generator=g) * 8, torch.rand(n, generator=g) * 24)
    py = torch.rand(n, generator=g) * 8
    depth = 3.0 - z
    # looking down -z: image x runs along +x, image y along -y
    pos = torch.stack([(px - 12) / 24 * depth, -(py - 8) / 24 * depth, z], dim=1).contiguous()
    opac = (torch.rand((n, 1), generator=g) * 0.9 + 0.1) * min(0.5, 40.0 / n)
    return view, pos, opac


# a tile's list is cut into segments of at least 256 instances; their length doubles from 655,360 instances on
@pytest.mark.parametrize("n", [1, 255, 256, 257, 511, 513, 769, 4097, 655_000, 700_001])
@pytest.mark.parametrize("rows", [0, 4, 16, 32])
@pytest.mark.parametrize("width, height", [(24, 16), (1040, 1024)])    # all tiles by two warps per list; more tiles than that, by one
def test_blend_at_the_edges_of_its_segments(n, rows, width, height):
    import inpc_b200
    from helpers import assert_close, oracle_camera
    if n > 100_000 and rows not in (0, 16):
        pytest.skip("the long lists are walked in one layout of each kind")
    view, pos, opac = _one_tile_scene(n, n, width, height)
    g = torch.Generator().manual_seed(n + 1)
    gi, ga = torch.randn((rows or 4, height, width), generator=g) * 1e-3, torch.randn((1, height, width), generator=g) * 1e-3
    cam, v, rast = oracle_camera(view), view.to(DEV), inpc_b200.INPCRasterizer()
    o = opac.to(DEV).requires_grad_(True)
    if rows:
        feats = torch.randn((n, rows), generator=g) * 0.5
        f = feats.to(DEV).requires_grad_(True)
        image, alpha, bw = rast.forward_rows(v, pos.to(DEV), f, o)
        st = O.rasterize_rows_forward(cam, pos.numpy(), feats.numpy(), opac.numpy())
        gf, go = O.rasterize_rows_backward(st, gi.numpy(), ga.numpy())
        tol_f = dict(rtol=2e-4, atol=1e-9)
    else:
        feats = (torch.randn((n, 36), generator=g) * 0.5).to(torch.float16)
        f = feats.to(DEV).requires_grad_(True)
        image, alpha, bw = rast(v, 0, pos.to(DEV), f, o)
        st = O.rasterize_forward(O.BILINEAR, cam, pos.numpy(), feats.numpy(), opac.numpy())
        gf, go, _ = O.rasterize_backward(st, gi.numpy(), ga.numpy())
        tol_f = dict(rtol=2e-3, atol=1.2e-7)      # two steps of the smallest halves
    # A pixel meets up to N = n / 16 fragments (four per point, three quarters of the points on 64 pixels).  Its transmittance is
    # a product of N factors; every product rounds by at most 2^-25, and while it is close to 1 mostly in the same direction, so
    # two orders of multiplication differ by up to N 2^-25 (measured against double precision: the oracle is off by 2.5e-5 for
    # n = 655,000, a tenth of the bound).  Everything else is proportional to it; sums of N terms add sqrt(N) 2^-24.
    eps = n / 16 * 2.0 ** -25
    assert_close(image.detach().cpu().numpy(), st.image, rtol=1e-4, atol=3e-6 + 0.2 * eps, what="image")
    assert_close(alpha.detach().cpu().numpy(), st.alpha, rtol=1e-5, atol=1e-6 + eps, what="alpha")
    assert_close(bw.cpu().numpy(), st.blending_weights, rtol=2e-4 + eps, atol=1e-9, what="blending weights")
    torch.autograd.backward([image, alpha], [gi.to(DEV), ga.to(DEV)])
    assert_close(f.grad.float().cpu().numpy(), np.asarray(gf, np.float32), rtol=tol_f["rtol"] + eps, atol=tol_f["atol"], what="grad_features")
    # opacity gradients are differences of sums of the order of 1e-3
    assert_close(o.grad.cpu().numpy(), go, rtol=1e-3 + eps, atol=2e-8 + 1e-3 * eps, what="grad_opacities")


# Opacities that are none: the products of later segments are sums of logarithms, which know no factor above one and no NaN by
# themselves.  A pixel whose transmittance is no number has no stop, and its alpha is no number.
@pytest.mark.parametrize("n", [700, 4097])
@pytest.mark.parametrize("odd", ["negative", "nan"])
@pytest.mark.parametrize("rows", [0, 8])
@pytest.mark.parametrize("width, height", [(24, 16), (1040, 1024)])    # all tiles by two warps per list; more tiles than that, by one
def test_odd_opacities_in_lists_of_several_segments(n, odd, rows, width, height):
    import inpc_b200
    from helpers import assert_close, oracle_camera
    view, pos, opac = _one_tile_scene(n, n, width, height)
    opac = opac.clone()
    if odd == "negative":
        opac[::9] *= -0.5
    else:
        opac[torch.argsort(3.0 - pos[:, 2])[n * 3 // 4]] = float("nan")     # behind the first segment of the tile it is in
    g = torch.Generator().manual_seed(n + 1)
    cam, v, rast = oracle_camera(view), view.to(DEV), inpc_b200.INPCRasterizer()
    if rows:
        feats = torch.randn((n, rows), generator=g) * 0.5
        image, alpha, bw = rast.forward_rows(v, pos.to(DEV), feats.to(DEV), opac.to(DEV))
        st = O.rasterize_rows_forward(cam, pos.numpy(), feats.numpy(), opac.numpy())
    else:
        feats = (torch.randn((n, 36), generator=g) * 0.5).to(torch.float16)
        image, alpha, bw = rast(v, 0, pos.to(DEV), feats.to(DEV), opac.to(DEV))
        st = O.rasterize_forward(O.BILINEAR, cam, pos.numpy(), feats.numpy(), opac.numpy())
        _, depth, inferred = rast.render_preextracted(v, 0, pos.to(DEV), feats.to(DEV), opac.to(DEV))
        _, odepth, oinferred, _ = O.render_preextracted(O.BILINEAR, cam, pos.numpy(), feats.numpy(), opac.numpy(), None, 0.05, 3.0)
        np.testing.assert_array_equal(np.isnan(inferred.cpu().numpy()), np.isnan(oinferred))
        np.testing.assert_array_equal(np.isnan(depth.cpu().numpy()), np.isnan(odepth))
        assert_close(inferred.cpu().numpy(), oinferred, rtol=1e-5, atol=1e-6 + n / 16 * 2.0 ** -25, what="alpha of inference")
    eps = n / 16 * 2.0 ** -25      # see the test of the segment edges
    for got, want, what in ((image, st.image, "image"), (alpha, st.alpha, "alpha"), (bw, st.blending_weights, "blending weights")):
        got = got.detach().cpu().numpy()
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want), err_msg=what)
        assert_close(got, want, rtol=2e-4 + eps, atol=3e-6 + eps, what=what)
    assert bool(np.isnan(st.alpha).any()) == (odd == "nan")


# A pixel whose colour is no number gives none to the opacities of all points it meets, before and behind the one at fault, and no feature gradient to
# those behind; the others are as they were.
@pytest.mark.parametrize("n", [1, 5, 40, 700, 4097])
@pytest.mark.parametrize("rows, tile", [(0, 8), (0, 16), (4, 8), (16, 8), (8, 16)])
@pytest.mark.parametrize("width, height", [(24, 16), (1040, 1024)])    # all tiles by two warps per list; more tiles than that, by one
def test_gradients_behind_an_opacity_that_is_no_number(n, rows, tile, width, height):
    import inpc_b200
    from helpers import assert_close, oracle_camera
    view, pos, opac = _one_tile_scene(n, n, width, height)
    opac = opac.clone()
    opac[torch.argsort(3.0 - pos[:, 2])[n * 3 // 4]] = float("nan")
    g = torch.Generator().manual_seed(n + 1)
    gi, ga = torch.randn((rows or 4, height, width), generator=g) * 1e-3, torch.randn((1, height, width), generator=g) * 1e-3
    cam, v, rast = oracle_camera(view), view.to(DEV), inpc_b200.INPCRasterizer(tile_size=tile)
    o = opac.to(DEV).requires_grad_(True)
    if rows:
        feats = torch.randn((n, rows), generator=g) * 0.5
        f = feats.to(DEV).requires_grad_(True)
        image, alpha, _ = rast.forward_rows(v, pos.to(DEV), f, o)
        gf, go = O.rasterize_rows_backward(O.rasterize_rows_forward(cam, pos.numpy(), feats.numpy(), opac.numpy()), gi.numpy(), ga.numpy())
    else:
        feats = (torch.randn((n, 36), generator=g) * 0.5).to(torch.float16)
        f = feats.to(DEV).requires_grad_(True)
        image, alpha, _ = rast(v, 0, pos.to(DEV), f, o)
        gf, go, _ = O.rasterize_backward(O.rasterize_forward(O.BILINEAR, cam, pos.numpy(), feats.numpy(), opac.numpy()), gi.numpy(), ga.numpy())
    torch.autograd.backward([image, alpha], [gi.to(DEV), ga.to(DEV)])
    assert np.isnan(go).any() and (n < 40 or not np.isnan(go).all())
    for got, want, tol, what in ((f.grad, gf, dict(rtol=2e-4, atol=1e-9) if rows else dict(rtol=2e-3, atol=1.2e-7), "features"),
                                 (o.grad, go, dict(rtol=1e-3, atol=2e-8), "opacities")):
        got, want = got.float().cpu().numpy(), np.asarray(want, np.float32)
        np.testing.assert_array_equal(np.isnan(got), np.isnan(want), err_msg=what)
        ok = ~np.isnan(want)
        eps = n / 16 * 2.0 ** -25      # see the test of the segment edges
        assert_close(got[ok], want[ok], rtol=tol["rtol"] + eps, atol=tol["atol"] + 1e-3 * eps, what=what)


# Where a pixel stops, its colour minus the running colour is zero to the bit, which 1 / (1 - alpha) would else multiply by up to 10^8:
# also where the opaque splat lies in a later segment.
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n_before", [100, 255, 256, 300, 511, 700, 1500])
@pytest.mark.parametrize("width, height", [(17, 9), (1033, 1025)])      # two warps per list; one
def test_opacity_gradient_of_an_opaque_splat_in_a_later_segment(mode, n_before, width, height):
    import inpc_b200
    from helpers import assert_close, oracle_camera
    from inpc_b200.views import look_at_view
    n, g = n_before + 20, torch.Generator().manual_seed(n_before)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, height, 16.0, 16.0, center_x=8.5, center_y=4.5)      # the axis meets the centre of pixel (8, 4)
    pos = torch.zeros((n, 3))
    pos[:, 2] = 1.0 - torch.arange(n) * 2.0 ** -11
    opac = torch.rand((n, 1), generator=g) * min(2e-3, 1.0 / n)
    opac[n_before] = 1.0
    feats = (torch.randn((n, 36), generator=g) * 0.5).to(torch.float16)
    gi, ga = torch.randn((4, height, width), generator=g) * 1e-3, torch.randn((1, height, width), generator=g) * 1e-3
    o = opac.to(DEV).requires_grad_(True)
    image, alpha, _ = inpc_b200.INPCRasterizer()(view.to(DEV), mode, pos.to(DEV), feats.to(DEV), o)
    torch.autograd.backward([image, alpha], [gi.to(DEV), ga.to(DEV)])
    st = O.rasterize_forward(mode, oracle_camera(view), pos.numpy(), feats.numpy(), opac.numpy())
    _, go, _ = O.rasterize_backward(st, gi.numpy(), ga.numpy())
    assert float(alpha.detach()[0, 4, 8]) == 1.0
    assert_close(o.grad.cpu().numpy(), go, rtol=1e-3, atol=2e-8, what="grad_opacities")


# A pixel whose transmittance comes to lie just above the stop still takes what is behind.  1 - alpha of an almost opaque splat depends on
# whether alpha has been rounded: by up to 2^-25, here 8.6e-5 of it, more than a pass may be early.  The splats lie in a later segment,
# the one behind them in the same or in the next.
@pytest.mark.parametrize("apart", [False, True])
@pytest.mark.parametrize("rows", [0, 8])
@pytest.mark.parametrize("width, height", [(64, 64), (1040, 1024)])     # two warps per list; one
def test_pixels_just_above_the_stop_in_a_later_segment(apart, rows, width, height):
    import inpc_b200
    from helpers import assert_close, oracle_camera
    from inpc_b200.views import look_at_view
    side, u, stop = 64, 2.0 ** -24, float(np.float32(1e-4))
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, height, float(side), float(side), center_x=side / 2, center_y=side / 2)
    cam = oracle_camera(view)

    def at(px, py, depth):
        z = torch.full_like(px, 3.0) - depth
        return torch.stack([(px - side / 2) / side * depth, -(py - side / 2) / side * depth, z], dim=1)
    c = torch.arange(0, side, 2, dtype=torch.float32) + 0.5
    py, px = (t.reshape(-1) for t in torch.meshgrid(c, c, indexing="ij"))           # every second pixel: no site reaches another
    t, dx = torch.arange(4, side, 8, dtype=torch.float32), 1.75e-4

    def clear(per_tile, depth):                                                      # splats of opacity zero
        ty, tx = (v.reshape(-1).repeat(per_tile) for v in torch.meshgrid(t, t, indexing="ij"))
        return at(tx, ty, depth)
    # in front of them a first segment of 256, between them a batch of 32 or another segment
    parts = [at(px + dx, py, 2.0), clear(300, 2.2), at(px + dx, py, 2.4), clear(300 if apart else 40, 2.5), at(px, py, 2.6)]
    first = np.cumsum([0] + [len(p) for p in parts])
    pos, n, m = torch.cat(parts).contiguous(), int(first[-1]), len(px)
    half = np.zeros((n, 36), np.float16)
    xy = O.preprocess_and_order(O.BILINEAR, O.TRAIN, cam, pos.numpy(), half, np.ones(n, np.float32)).screen.reshape(-1, 2)
    one, centre = np.float32(1), np.stack([px.numpy(), py.numpy()], axis=1)

    def weight(part):
        d = one - np.abs(xy[first[part]:first[part] + m] - centre)
        return d[:, 0] * d[:, 1]
    w0, w1 = weight(0), weight(2)
    b = np.round((1.0 - w1.astype(np.float64)) / u)
    opac1 = (1.0 - np.round(0.497 / u / b) * u).astype(np.float32)                   # the product of two such factors ends halfway between two floats
    rounded, exact = (one - opac1 * w1).astype(np.float64), 1.0 - opac1.astype(np.float64) * w1
    opac0 = ((1.0 - stop / rounded * (1.0 + 4e-6)) / w0).astype(np.float32)
    left = (one - opac0 * w0).astype(np.float64)
    assert (left * rounded > stop * (1 + 2e-6)).all() and (left * exact < stop * (1 - 7.5e-5)).all()
    opac = np.zeros((n, 1), np.float32)
    opac[:m, 0], opac[first[2]:first[2] + m, 0], opac[n - m:, 0] = opac0, opac1, 1.0
    rast, v, p, o = inpc_b200.INPCRasterizer(), view.to(DEV), pos.to(DEV), torch.from_numpy(opac).to(DEV)
    if rows:
        feats = np.zeros((n, rows), np.float32)
        feats[n - m:] = 1e4
        st = O.rasterize_rows_forward(cam, pos.numpy(), feats, opac)
        image, alpha, bw = rast.forward_rows(v, p, torch.from_numpy(feats).to(DEV), o)
    else:
        half[n - m:, :4] = 2e4
        st = O.rasterize_forward(O.BILINEAR, cam, pos.numpy(), half, opac)
        image, alpha, bw = rast(v, 0, p, torch.from_numpy(half).to(DEV), o)
    sites = np.s_[:, 0:side:2, 0:side:2]
    assert (st.image[sites] > 0.2).all()                                             # a ten-thousandth of what the last splats hold
    # the transmittance is 1 - alpha with alpha of almost 1: a rounding of the opacity's product is 2^-24 / 3.4e-4
    assert_close(image.cpu().numpy()[sites], st.image[sites], rtol=4e-4, what="image")
    assert_close(bw.cpu().numpy()[n - m:], st.blending_weights[n - m:], rtol=4e-4, what="blending weights")
    assert float(alpha.min()) >= 0.0 and bool((alpha[sites] == 1.0).all())


# The same over all blends, against the same splats in a list of one segment: clear splats between them do not move a pixel's stop.  The
# opacities are chosen from what an almost opaque splat alone leaves, so that a pixel's transmittance lies within 10^-4 of the stop on either side.
@pytest.mark.parametrize("inference", [False, True])
@pytest.mark.parametrize("mode,tile", [(0, 8), (0, 16), (1, 8), (1, 16)])
@pytest.mark.parametrize("width, height", [(64, 64), (1040, 1024)])     # two warps per list; one
def test_clear_splats_do_not_move_the_stop(mode, tile, inference, width, height):
    import inpc_b200
    from inpc_b200.views import look_at_view
    side, clear, trials = 64, 300 if tile == 8 else 6000, 8          # a first segment has 256 or 4096 instances here
    v = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, height, float(side), float(side), center_x=side / 2, center_y=side / 2).to(DEV)
    rast, g = inpc_b200.INPCRasterizer(tile_size=tile), torch.Generator().manual_seed(tile + mode)

    def at(px, py, depth):
        return torch.stack([(px - side / 2) / side * depth, -(py - side / 2) / side * depth, torch.full_like(px, 3.0) - depth], dim=1)

    def blend(parts, opacities, lit):
        pos, n = torch.cat(parts).contiguous().to(DEV), sum(len(p) for p in parts)
        feats = torch.zeros((n, 36), dtype=torch.float16)
        feats[n - lit:, :4] = 2e4
        opac = torch.cat(opacities).reshape(-1, 1).contiguous().to(DEV)
        out = rast.render_preextracted(v, mode, pos, feats.to(DEV), opac) if inference else rast(v, mode, pos, feats.to(DEV), opac)
        return out[0][0, 1:side:4, 1:side:4].cpu().reshape(-1), out[2 if inference else 1][0, 1:side:4, 1:side:4].cpu().double().reshape(-1)
    c, t = torch.arange(1, side, 4, dtype=torch.float32) + 0.5, torch.arange(tile / 2, side, tile)
    py, px = (x.reshape(-1) for x in torch.meshgrid(c, c, indexing="ij"))
    ty, tx = (x.reshape(-1).repeat(clear) for x in torch.meshgrid(t, t, indexing="ij"))
    m, moved, lit = len(px), 0, 0
    for _ in range(trials):
        dx = torch.rand(m, generator=g) * (2e-4 if mode == 0 else 0.02)
        o1 = 1.0 - 10.0 ** (torch.rand(m, generator=g) * 0.6 - 3.7)
        splats, none = [at(px, py, 2.0), at(px + dx, py, 2.4), at(px, py, 2.6)], torch.zeros(len(tx))
        left = 1.0 - blend(splats[1:2], [o1], 0)[1]
        o0 = (1.0 - 1e-4 / left * (1.0 + (torch.rand(m, generator=g).double() * 2 - 1) * 1e-4)).float()
        o2 = torch.ones(m)
        one = blend(splats, [o0, o1, o2], m)[0]
        many = blend([splats[0], at(tx, ty, 2.2), splats[1], at(tx, ty, 2.5), splats[2]], [o0, none, o1, none, o2], m)[0]
        moved += int(((one > 0.1) != (many > 0.1)).sum())            # the last splats add 0.56 where a pixel is still open
        lit += int((one > 0.1).sum())
    # two orders of multiplying and adding up four factors are up to 2^-22 apart, of a range of 2 * 10^-4: one pixel in 420 on either side
    assert 0.2 * m * trials < lit < 0.8 * m * trials and moved <= m * trials / 200, (moved, lit, m * trials)


# Lists of several segments of very faint splats: the segments' transmittances come from sums of logarithms, which may be no
# further from double precision than the chain of fp32 products the oracle forms.
@pytest.mark.parametrize("n,opacity", [(40_000, 2e-6), (200_000, 2e-6), (200_000, 2e-5)])
@pytest.mark.parametrize("width, height", [(96, 64), (1040, 1024)])     # two warps per list; one
def test_faint_splats_are_as_exact_as_a_chain_of_products(n, opacity, width, height):
    from dataclasses import replace
    import inpc_b200
    from helpers import oracle_camera, small_scene
    from inpc_b200.views import View
    view, pos, feats, opac = small_scene(n=n, width=96, height=64, focal=82.0)
    opac = (opac * opacity).contiguous()
    view = View(replace(view.camera, width=width, height=height), view.w2c, view.position)      # (the same pixels in its upper left corner)
    _, alpha, _ = inpc_b200.INPCRasterizer()(view.to(DEV), 0, pos.to(DEV), feats.to(DEV), opac.to(DEV))
    st = O.rasterize_forward(O.BILINEAR, oracle_camera(view), pos.numpy(), feats.numpy(), opac.numpy())
    # double precision: -log of the product over the 2x2 pixels of every visible point
    seen = np.unique(st.inst_point)
    xy, op = st.screen.reshape(-1, 2)[seen].astype(np.float64), opac.numpy().reshape(-1)[seen].astype(np.float64)
    total, base = np.zeros((64, 96)), np.floor(xy - 0.5).astype(np.int64)
    for dx in (0, 1):
        for dy in (0, 1):
            px, py = base[:, 0] + dx, base[:, 1] + dy
            w = np.clip(1 - np.abs(xy[:, 0] - px - 0.5), 0, 1) * np.clip(1 - np.abs(xy[:, 1] - py - 0.5), 0, 1)
            ok = (px >= 0) & (px < 96) & (py >= 0) & (py < 64)
            np.add.at(total, (py[ok], px[ok]), np.log1p(-op[ok] * w[ok]))
    exact = -np.expm1(total)
    off = [np.sqrt(((a.reshape(height, width)[:64, :96].astype(np.float64) - exact) ** 2).mean()) for a in (alpha.cpu().numpy(), st.alpha)]
    assert off[0] <= 1.25 * off[1], off


# gaussian splats on 8x8 tiles: footprints from a fraction of a pixel to several tiles, image sides around tile and half borders
@pytest.mark.parametrize("width,height", [(8, 4), (9, 5), (64, 36), (67, 45)])
@pytest.mark.parametrize("sigma_px", [0.01, 0.7, 3.0, 40.0])
def test_gaussian_footprints_at_tile_edges(width, height, sigma_px):
    import inpc_b200
    from helpers import assert_close, oracle_camera
    from inpc_b200.views import look_at_view
    g = torch.Generator().manual_seed(width * 7 + int(sigma_px * 100))
    n, focal = 300, 0.5 * width                     # a wide view: splats off the axis are long ellipses
    view = look_at_view((0.1, 0.2, 2.0), (0.0, 0.0, 0.0), width, height, focal, focal * 1.1)
    pos = ((torch.rand((n, 3), generator=g) * 2 - 1) * torch.tensor([2.5, 2.0, 1.2])).contiguous()
    feats = (torch.randn((n, 36), generator=g) * 0.5).to(torch.float16)
    opac = torch.rand((n, 1), generator=g) * 0.3 + 0.01
    scales = torch.exp(torch.randn((n, 1), generator=g) * 0.5) * (2.0 * sigma_px / focal)
    img, dep, alp = inpc_b200.INPCRasterizer().render_preextracted(view.to(DEV), 1, pos.to(DEV), feats.to(DEV), opac.to(DEV), scales.to(DEV))
    oi, od, oa, _ = O.render_preextracted(O.GAUSSIAN, oracle_camera(view), pos.numpy(), feats.numpy(), opac.numpy(), scales.numpy(),
                                          0.05 / view.camera.focal_y, 3.0)
    # a fragment within rounding of the cut-off (weight 0.011 of at most 0.31) may fall on either side of it
    for got, want, what in ((img, oi, "image"), (dep, od, "depth"), (alp, oa, "alpha")):
        assert_close(got.cpu().numpy(), want, rtol=2e-4, atol=2e-5, max_bad=4, what=what)


def _clear_of_the_cutoff(st, pos, threshold, reach):
    """The points, those behind the camera whose weight at some pixel within `reach` lies so close to the threshold that rounding
    (two units of the last place of the exponential, and of its argument) decides on which side it falls."""
    xy, c = st.screen.reshape(-1, 2).astype(np.float64), st.conic.reshape(-1, 3).astype(np.float64)
    near = np.zeros(len(xy), bool)
    base = np.floor(xy) + 0.5
    for ox in range(-reach, reach + 1):
        for oy in range(-reach, reach + 1):
            dx, dy = xy[:, 0] - base[:, 0] - ox, xy[:, 1] - base[:, 1] - oy
            q = -0.5 * (c[:, 0] * dx * dx + c[:, 2] * dy * dy) - c[:, 1] * dx * dy
            near |= np.abs(q - np.log(threshold)) < 1e-4
    out = pos.clone()
    out[torch.from_numpy(near)] = torch.tensor([0.0, 0.0, 10.0])
    return out, int(near.sum())


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 513, 20_001, 700_001])
@pytest.mark.parametrize("width, height", [(24, 16), (1040, 1024)])    # all tiles by two warps per list; more tiles than that, by one
def test_gaussian_blend_at_the_edges_of_its_segments(n, width, height):
    import inpc_b200
    from helpers import assert_close, oracle_camera
    view, pos, opac = _one_tile_scene(n, n, width, height)
    cam = oracle_camera(view)
    g = torch.Generator().manual_seed(n + 1)
    gi, ga = torch.randn((4, height, width), generator=g) * 1e-3, torch.randn((1, height, width), generator=g) * 1e-3
    feats = (torch.randn((n, 36), generator=g) * 0.5).to(torch.float16)
    pos, dropped = _clear_of_the_cutoff(O.preprocess_and_order(O.GAUSSIAN, O.TRAIN, cam, pos.numpy(), feats.numpy(), opac.numpy()), pos,
                                        0.01110899653, 3)
    assert dropped <= n // 200
    f, o = feats.to(DEV).requires_grad_(True), opac.to(DEV).requires_grad_(True)
    image, alpha, bw = inpc_b200.INPCRasterizer()(view.to(DEV), 1, pos.to(DEV), f, o)
    st = O.rasterize_forward(O.GAUSSIAN, cam, pos.numpy(), feats.numpy(), opac.numpy())
    gf, go, _ = O.rasterize_backward(st, gi.numpy(), ga.numpy())
    torch.autograd.backward([image, alpha], [gi.to(DEV), ga.to(DEV)])
    # the bounds of the bilinear test with about six fragments per point; the exponentials of device and oracle differ by two
    # units of the last place
    eps = n / 10 * 2.0 ** -25 + 2.0 ** -22
    assert_close(image.detach().cpu().numpy(), st.image, rtol=1e-4, atol=1e-5 + 0.2 * eps, what="image")
    assert_close(alpha.detach().cpu().numpy(), st.alpha, rtol=1e-5, atol=1e-6 + eps, what="alpha")
    assert_close(bw.cpu().numpy(), st.blending_weights, rtol=4e-4 + eps, atol=1e-9, what="blending weights")
    assert_close(f.grad.float().cpu().numpy(), np.asarray(gf, np.float32), rtol=4e-3 + eps, atol=2e-7, what="grad_features")
    assert_close(o.grad.cpu().numpy(), go, rtol=2e-3 + eps, atol=4e-8 + 1e-3 * eps, what="grad_opacities")
    assert all(bool(torch.isfinite(t).all()) for t in (image, alpha, bw, f.grad, o.grad))


# inference with a size per splat over lists of several segments: the depth and the transmittance at which a pixel stopped come from
# the segments' own
@pytest.mark.parametrize("n", [255, 257, 1023, 4097, 20_001])
@pytest.mark.parametrize("strength", [0.1, 1.0, 30.0])
def test_gaussian_inference_over_several_segments(n, strength):
    import inpc_b200
    from helpers import assert_close, oracle_camera
    view, pos, opac = _one_tile_scene(n, n)
    opac, cam = (opac * strength).clamp(max=0.9).contiguous(), oracle_camera(view)
    g = torch.Generator().manual_seed(n + 2)
    feats = (torch.randn((n, 36), generator=g) * 0.5).to(torch.float16)
    scales = torch.exp(torch.randn((n, 1), generator=g) * 0.4) * 0.06          # about one and a half pixels
    sigma = inpc_b200.INPCRasterizer.extract_base_sigma_world(view.camera)

    def oracle(p):
        return O.render_preextracted(O.GAUSSIAN, cam, p.numpy(), feats.numpy(), opac.numpy(), scales.numpy(), sigma, 3.0)
    pos, dropped = _clear_of_the_cutoff(oracle(pos)[3], pos, np.exp(-4.5), 12)
    assert dropped <= n // 10
    image, depth, alpha = inpc_b200.INPCRasterizer().render_preextracted(view.to(DEV), 1, pos.to(DEV), feats.to(DEV), opac.to(DEV), scales.to(DEV))
    oi, od, oa, _ = oracle(pos)
    # inference takes the fast exponential: off by 2 + 1.2 |q| units of the last place, |q| <= 4.5; some 25 fragments per point.  A
    # pixel within rounding of its stop may take a fragment more or less: up to 10^-4 of its transmittance, where pixels stop at all.
    stop = 1.1e-4 if float(oa.max()) == 1.0 else 0.0
    eps = n * 2.0 ** -25 + 2.0 ** -21
    assert_close(image.cpu().numpy(), oi, rtol=1e-4, atol=1e-5 + 0.2 * eps + stop, what="image")
    assert_close(alpha.cpu().numpy(), oa, rtol=1e-5, atol=1e-6 + eps + stop, what="alpha")
    some = oa[0] > 1e-2            # the depth divides by alpha
    assert_close(depth.cpu().numpy()[0][some], od[0][some], rtol=1e-4 + 100 * eps + stop, what="depth")
    assert all(bool(torch.isfinite(t).all()) for t in (image, depth, alpha))


# four points per thread and 16-byte loads where the positions are aligned; one block gathers 256 points
@pytest.mark.parametrize("n", [1, 2, 3, 5, 255, 257, 1023, 1025, 300_001])
@pytest.mark.parametrize("offset", [0, 1])
def test_morton_order_at_block_edges_and_offsets(n, offset):
    from inpc_b200.sampling import morton_order
    g = torch.Generator().manual_seed(n)
    pos = (torch.rand((n + offset, 3), generator=g) * torch.tensor([2.0, 1.0, 3.0]) - 1.0)[offset:]     # offset 1: rows start 12 bytes on
    lo = pos.min(dim=0).values
    extent = float((pos.max(dim=0).values - lo).max())
    inv = np.float32(1.0) / np.float32(np.float64(extent) * (1.0 + 1e-6)) if extent > 0 else np.float32(1.0)
    q = ((pos - lo) * torch.tensor(inv) * 1024.0).clamp(0.0, 1023.0).to(torch.int64)
    code = sum((((q[:, c] >> b) & 1) << (3 * b + c)) for b in range(10) for c in range(3))
    store = torch.empty((n + offset, 3), device=DEV)
    src = store[offset:]
    src.copy_(pos)
    assert torch.equal(morton_order(src).cpu(), pos[torch.sort(code, stable=True).indices])


# a NaN leaves its axis without a corner (its part of the codes is zero) and the cube with an edge of 1; infinities are ordinary values
@pytest.mark.parametrize("n", [2, 5, 257, 4099, 300_001])
@pytest.mark.parametrize("odd", ["one_nan", "nan_axis", "nan_rows", "inf", "minus_inf"])
def test_morton_order_of_clouds_with_odd_coordinates(n, odd):
    from inpc_b200.sampling import morton_order
    g = torch.Generator().manual_seed(n)
    pos = torch.rand((n, 3), generator=g) * torch.tensor([2.0, 1.0, 3.0]) - 1.0
    if odd == "one_nan":
        pos[n // 2, 2] = float("nan")
    elif odd == "nan_axis":
        pos[::3, 1] = float("nan")
    elif odd == "nan_rows":
        pos[::4] = float("nan")
    else:
        pos[n - 1, 0] = float("inf") if odd == "inf" else -float("inf")
    lo = pos.amin(dim=0)
    extent = float((pos.amax(dim=0) - lo).max())
    inv = np.float32(1.0) / np.float32(np.float64(extent) * (1.0 + 1e-6)) if extent > 0 else np.float32(1.0)
    q = ((pos - lo) * torch.tensor(inv) * 1024.0).nan_to_num(nan=0.0).clamp(0.0, 1023.0).to(torch.int64)
    code = sum((((q[:, c] >> b) & 1) << (3 * b + c)) for b in range(10) for c in range(3))
    want = pos[torch.sort(code, stable=True).indices]
    assert torch.equal(morton_order(pos.to(DEV)).cpu().view(torch.int32), want.view(torch.int32))
