"""GPU tests of the walk backward through short lists: every fragment of a list in the same one to four pixels, at the edges of the chunks
and batches it is walked in and of the halves and tiles a footprint can straddle, against 64-bit arithmetic."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SIDE = 24


U = 2.0 ** -24      # largest relative error of a rounding to 32 bits


def _exact(x, y, opacity, features, grad_image, grad_alpha):
    """Gradients of opacities and features of splats at (x, y) (front to back) in 64 bits, and how far 32-bit arithmetic may be off, per
    splat: every operation rounds by U of its result, and what a fragment meets or leaves behind carries the errors of the fragments before it."""
    go, gf = np.zeros(len(x)), np.zeros(features.shape)
    go_bound, gf_bound = np.zeros(len(x)), np.zeros(features.shape)
    channels = features.shape[1]
    for row in range(SIDE):
        for column in range(SIDE):
            w = np.clip(1 - np.abs(x - (column + 0.5)), 0, 1) * np.clip(1 - np.abs(y - (row + 0.5)), 0, 1)
            k = np.nonzero(w > 0)[0]
            if len(k) == 0:
                continue
            al = opacity[k] * w[k]
            met = np.cumprod(np.concatenate([[1.0], 1 - al]))
            stop = np.nonzero(met[1:] < 1e-4)[0]
            m = int(stop[0]) + 1 if len(stop) else len(k)
            k, al, T, end = k[:m], al[:m], met[:m], met[m]
            g = grad_image[:, row, column]
            G, bw = features[k] @ g, T * al
            behind = (bw * G).sum() - np.cumsum(bw * G)
            upstream = 0.0 if len(stop) else grad_alpha[0, row, column]
            K = upstream * end
            go[k] += (T * G + (K - behind) / np.maximum(1 - al, 1e-8)) * w[k]
            gf[k] += bw[:, None] * g[None]
            # alpha is off by 4 U of itself (weight: two differences, two products), a transmittance by that over one minus alpha, and by two
            # roundings, of every fragment before
            off_T = np.concatenate([[0.0], np.cumsum((4 * al / (1 - al) + 2) * U)])
            G_abs = np.abs(features[k]) @ np.abs(g)
            sum_abs = (bw * G_abs).sum()
            off_behind = (bw * G_abs * (off_T[:m] + (channels + 6) * U)).sum() + 2 * (m + channels) * U * sum_abs   # two running sums of m terms
            off_K = np.abs(upstream) * (end * off_T[m] + 2 * U)
            go_bound[k] += w[k] * (T * G_abs * (off_T[:m] + (channels + 6) * U) +
                                   (off_behind + off_K + np.abs(K - behind) * (6 + 4 * al / (1 - al)) * U) / (1 - al))
            gf_bound[k] += bw[:, None] * np.abs(g)[None] * (off_T[:m, None] + 8 * U)
    return go, gf, go_bound, gf_bound


def _sh_basis(position, eye):
    x, y, z = ((position - eye) / np.linalg.norm(position - eye, axis=1, keepdims=True)).T
    return np.stack([np.full_like(x, 0.28209479177387814), -0.48860251190291987 * y, 0.48860251190291987 * z, -0.48860251190291987 * x, 1.0925484305920792 * x * y,
                     -1.0925484305920792 * y * z, 0.94617469575755997 * z * z - 0.31539156525251999, -1.0925484305920792 * x * z,
                     0.54627421529603959 * (x * x - y * y)], axis=1)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 9, 31, 32, 33, 65])
@pytest.mark.parametrize("opaque", [False, True])
@pytest.mark.parametrize("site", [(7.0, 3.0), (8.0, 4.0), (8.0, 8.0), (12.0, 10.0), (13.0, 5.0), (0.25, 0.25), (23.75, 23.75)])
def test_lists_of_one_footprint(n, opaque, site):
    import inpc_b200
    from inpc_b200 import rasterization as R
    from inpc_b200.views import look_at_view
    g = torch.Generator().manual_seed(n * 2 + opaque)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), SIDE, SIDE, float(SIDE), float(SIDE)).to(DEV)
    depth = 2.0 + 0.01 * torch.arange(n, dtype=torch.float32)
    px, py = site[0] + (torch.rand(n, generator=g) - 0.5) * 0.8, site[1] + (torch.rand(n, generator=g) - 0.5) * 0.8
    pos = torch.stack([(px - SIDE / 2) / SIDE * depth, -(py - SIDE / 2) / SIDE * depth, 3.0 - depth], dim=1).contiguous().to(DEV)
    opacity = torch.rand((n, 1), generator=g) * (0.2 if n < 32 else 0.05)
    if opaque:
        opacity[n // 2] = 0.999       # in a pixel close to its centre most of what is left ends here
    gi, ga = torch.randn((4, SIDE, SIDE), generator=g), torch.randn((1, SIDE, SIDE), generator=g)
    rast, settings = inpc_b200.INPCRasterizer(tile_size=8), R.INPCRasterizer.extract_settings(view, 0)
    sh = (torch.randn((n, 36), generator=g) * 0.5).to(torch.float16).to(DEV)
    _, _, _, state, blobs, _ = R.forward_with_state(pos, sh, opacity.to(DEV), settings, 8)
    dbg = R.debug_arrays(state, settings, blobs.point, blobs.instance)
    x, y = dbg["screen"].double().cpu().numpy().T
    assert int(state.n_visible) == n
    for rows in (0, 4, 16):
        features = torch.randn((n, rows), generator=g).to(DEV) if rows else sh
        f, o = features.requires_grad_(True), opacity.to(DEV).requires_grad_(True)
        image, alpha, _ = rast.forward_rows(view, pos, f, o) if rows else rast(view, 0, pos, f, o)
        gi_c = gi if rows != 16 else gi.repeat(4, 1, 1)
        torch.autograd.backward([image, alpha], [gi_c.to(DEV), ga.to(DEV)])
        seen = (f.detach() if rows else dbg["feat_view"]).double().cpu().numpy()
        go, gf, go_bound, gf_bound = _exact(x, y, opacity.double().numpy()[:, 0], seen, gi_c.double().numpy(), ga.double().numpy())
        off = np.abs(o.grad.double().cpu().numpy()[:, 0] - go)
        assert (off <= go_bound).all(), (rows, (off / go_bound).max())
        if not rows:   # through the basis, and to halves: 2^-11 of the value, or half a step of the smallest ones
            basis = _sh_basis(pos.double().cpu().numpy(), np.array([0.0, 0.0, 3.0]))
            gf, gf_bound = ((basis[:, :, None] * v[:, None, :]).reshape(n, 36) for v in (gf, gf_bound))
            gf_bound = np.abs(gf_bound) + np.abs(gf) * 2.0 ** -11 + 2.0 ** -25 + 32 * U * np.abs(gf).max(axis=1, keepdims=True)
        off = np.abs(f.grad.double().cpu().numpy() - gf)
        assert (off <= gf_bound + 1e-30).all(), (rows, (off / (gf_bound + 1e-30)).max())


# Lists of many segments (of 256 instances each, so few are there): the transmittances at their starts are formed 16 at a time, by whichever segment is through last
@pytest.mark.parametrize("segments", [2, 3, 4, 16, 17, 18, 19, 33, 50])
@pytest.mark.parametrize("opaque", [False, True])
def test_lists_of_many_segments(segments, opaque):
    import inpc_b200
    from inpc_b200 import rasterization as R
    from inpc_b200.views import look_at_view
    n = 256 * segments - 100
    g = torch.Generator().manual_seed(segments * 2 + opaque)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), SIDE, SIDE, float(SIDE), float(SIDE)).to(DEV)
    depth = 2.0 + torch.arange(n, dtype=torch.float32) / 1024
    px, py = 9.0 + torch.rand(n, generator=g) * 6, 9.0 + torch.rand(n, generator=g) * 6   # inside the second tile in both directions
    pos = torch.stack([(px - SIDE / 2) / SIDE * depth, -(py - SIDE / 2) / SIDE * depth, 3.0 - depth], dim=1).contiguous().to(DEV)
    opacity = torch.rand((n, 1), generator=g) * (4.0 / n)          # in a pixel about a tenth of them: most of what is behind is seen
    if opaque:
        opacity[torch.arange(n) % 256 == 255] = 0.3                # a pixel stops in the middle of the list, at another place for each
    gi, ga = torch.randn((4, SIDE, SIDE), generator=g), torch.randn((1, SIDE, SIDE), generator=g)
    rast, settings = inpc_b200.INPCRasterizer(tile_size=8), R.INPCRasterizer.extract_settings(view, 0)
    sh = (torch.randn((n, 36), generator=g) * 0.5).to(torch.float16).to(DEV)
    _, _, _, state, blobs, _ = R.forward_with_state(pos, sh, opacity.to(DEV), settings, 8)
    dbg = R.debug_arrays(state, settings, blobs.point, blobs.instance)
    x, y = dbg["screen"].double().cpu().numpy().T
    assert int(state.n_visible) == n == int(state.n_instances)
    for rows in (0, 4, 16):
        features = torch.randn((n, rows), generator=g).to(DEV) if rows else sh
        f, o = features.requires_grad_(True), opacity.to(DEV).requires_grad_(True)
        image, alpha, _ = rast.forward_rows(view, pos, f, o) if rows else rast(view, 0, pos, f, o)
        gi_c = gi if rows != 16 else gi.repeat(4, 1, 1)
        torch.autograd.backward([image, alpha], [gi_c.to(DEV), ga.to(DEV)])
        seen = (f.detach() if rows else dbg["feat_view"]).double().cpu().numpy()
        go, gf, go_bound, gf_bound = _exact(x, y, opacity.double().numpy()[:, 0], seen, gi_c.double().numpy(), ga.double().numpy())
        off = np.abs(o.grad.double().cpu().numpy()[:, 0] - go)
        assert (off <= go_bound).all(), (rows, (off / go_bound).max())
        if rows:
            off = np.abs(f.grad.double().cpu().numpy() - gf)
            assert (off <= gf_bound + 1e-30).all(), (rows, (off / (gf_bound + 1e-30)).max())
    # gaussian splats, and inference of both: nothing depends on the tile size but the order of the sums
    feats, opac = sh.detach(), opacity.to(DEV)
    for mode in (0, 1):
        out = []
        for tile in (8, 16):
            f, o = feats.clone().requires_grad_(True), opac.clone().requires_grad_(True)
            r = inpc_b200.INPCRasterizer(tile_size=tile)
            image, alpha, weights = r(view, mode, pos, f, o)
            torch.autograd.backward([image, alpha], [gi.to(DEV), ga.to(DEV)])
            out.append((image.detach(), alpha.detach(), weights, o.grad, f.grad.float(), *r.render_preextracted(view, mode, pos, feats, opac)))
        for a, b in zip(*out):
            # products of up to n factors in another grouping, twice (their terms' transmittance and the stop)
            assert float((a - b).norm()) <= max(1e-4, 2 * n * U) * float(b.norm())


# Two warps per list (images of few tiles) against one: the same points in the upper left corner of an image that has more tiles than that.  Lists of every length beside a batch of 32, of
# faint splats, of which nothing stops, and of opaque ones, where the pixels stop in the middle of a batch, at its end, and one after the other
@pytest.mark.parametrize("opacity", [0.004, 0.3, 0.97, None])
@pytest.mark.parametrize("channels, mode", [(None, 0), (4, 0), (8, 0), (16, 0), (32, 0), (None, 1)])
def test_lists_walked_by_two_warps_and_by_one(channels, mode, opacity):
    import inpc_b200
    from inpc_b200.views import look_at_view
    width, height = 128, 16
    lengths = torch.tensor([1, 2, 31, 32, 33, 63, 64, 65, 66, 95, 96, 97, 98, 127, 128, 129, 160, 161, 192, 200, 223, 224, 225, 240, 250, 254, 255, 256, 0, 3, 48, 80])
    g = torch.Generator().manual_seed(channels or 0)
    n = int(lengths.sum())
    tile = torch.repeat_interleave(torch.arange(lengths.numel()), lengths)
    px, py = (tile % 16) * 8 + torch.rand(n, generator=g) * 6 + 1, (tile // 16) * 8 + torch.rand(n, generator=g) * 6 + 1
    z = torch.rand(n, generator=g)
    pos = torch.stack([(px - 64) / 64 * (3 - z), -(py - 8) / 64 * (3 - z), z], dim=1)[torch.randperm(n, generator=g)].contiguous().to(DEV)
    opac = (torch.rand((n, 1), generator=g) if opacity is None else torch.full((n, 1), opacity)).to(DEV)
    feats = torch.randn((n, channels or 36), generator=g).to(DEV)
    feats = feats if channels else (feats * 0.5).half()
    gi, ga = torch.randn((channels or 4, height, width), generator=g).to(DEV), torch.randn((1, height, width), generator=g).to(DEV)
    out = []
    for w, h in ((width, height), (4096, 520)):
        view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), w, h, 64.0, 64.0, center_x=64.0, center_y=8.0).to(DEV)
        f, o = feats.clone().requires_grad_(True), opac.clone().requires_grad_(True)
        rast = inpc_b200.INPCRasterizer()
        image, alpha, weights = rast.forward_rows(view, pos, f, o) if channels else rast(view, mode, pos, f, o)
        torch.autograd.backward([image[:, :height, :width], alpha[:, :height, :width]], [gi, ga])
        out.append((image[:, :height, :width].detach(), alpha[:, :height, :width].detach(), weights, f.grad, o.grad))
    assert int((out[0][1] > 0).sum()) > 500
    for k, (a, b) in enumerate(zip(*out)):
        # images and alphas to the bit, and the gradients of four channels, which have one writer each; the others are sums of up to four atomic additions in any order
        if k < 2 or (k > 2 and channels is None and mode == 0):
            assert torch.equal(a, b), k
        else:
            step = 2.0 ** -11 if k == 3 and mode == 1 else 8 * 2.0 ** -24       # (feature gradients of gaussian splats: a step of a half)
            assert float((a.float() - b.float()).abs().max()) <= step * float(torch.maximum(a.abs(), b.abs()).max()), k
