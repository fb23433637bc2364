"""GPU tests of the walk backward through short lists: every fragment of a list in the same one to four pixels, at the edges of the chunks
and batches it is walked in and of the halves and tiles a footprint can straddle, against 64-bit arithmetic."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SIDE = 24


def _exact(x, y, opacity, features, grad_image, grad_alpha):
    """Gradients of opacities and features of splats at (x, y) (front to back) in 64 bits."""
    go, gf = np.zeros(len(x)), np.zeros(features.shape)
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
            k, al, T = k[:m], al[:m], met[:m]
            g = grad_image[:, row, column]
            G, bw = features[k] @ g, T * al
            behind = (bw * G).sum() - np.cumsum(bw * G)
            K = 0.0 if len(stop) else grad_alpha[0, row, column] * met[m]
            go[k] += (T * G + (K - behind) / np.maximum(1 - al, 1e-8)) * w[k]
            gf[k] += bw[:, None] * g[None]
    return go, gf


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
        go, gf = _exact(x, y, opacity.double().numpy()[:, 0], seen, gi_c.double().numpy(), ga.double().numpy())
        # sums of up to n terms of order one, rounded by 2^-24 each; what lies behind a fragment is divided by its 1 - alpha, at least
        # 10^-3, times a transmittance of at least 10^-4 where the list does not end: sqrt(n) 2^-24 / (1 - alpha) of the largest gradient
        bound = (8 + np.sqrt(n)) * 2.0 ** -24 * (1e3 if opaque else 1.0) * max(1.0, np.abs(gi_c.numpy()).max()) * (1 + rows)
        np.testing.assert_allclose(o.grad.double().cpu().numpy()[:, 0], go, rtol=1e-4, atol=bound)
        if rows:
            np.testing.assert_allclose(f.grad.double().cpu().numpy(), gf, rtol=1e-5, atol=(8 + np.sqrt(n)) * 2.0 ** -24)
