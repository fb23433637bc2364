"""GPU tests of the order of points of which some are culled: they keep their place among the keys of the depth sort, whose first pass leaves
them out.  Counts, order, lists and ranges bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _scene(n, seen, seed, near=0.01, far=100.0):
    """n points of which `seen` (a mask) lie in front of a 40x24 image, the others behind the camera or beside it."""
    from inpc_b200.views import look_at_view
    g = torch.Generator().manual_seed(seed)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 40, 24, 40.0, 40.0, near_plane=near, far_plane=far)
    z = torch.rand(n, generator=g) * 1.5
    depth = 3.0 - z
    px, py = torch.rand(n, generator=g) * 40, torch.rand(n, generator=g) * 24
    pos = torch.stack([(px - 20) / 40 * depth, -(py - 12) / 40 * depth, z], dim=1)
    beside = torch.rand(n, generator=g) < 0.5
    hidden = torch.where(beside[:, None], pos + torch.tensor([50.0, 0.0, 0.0]), pos + torch.tensor([0.0, 0.0, 9.0]))
    return view, torch.where(seen[:, None], pos, hidden).contiguous(), torch.full((n, 1), 0.01)


def _check(view, pos, opac):
    from helpers import oracle_camera
    from inpc_b200 import rasterization as R
    n = pos.shape[0]
    v = view.to(DEV)
    settings = R.INPCRasterizer.extract_settings(v, 0)
    feats = torch.zeros((n, 36), dtype=torch.float16)
    _, _, _, state, blobs, _ = R.forward_with_state(pos.to(DEV), feats.to(DEV), opac.to(DEV), settings, 8)
    st = O.preprocess_and_order(O.BILINEAR, O.TRAIN, oracle_camera(view), pos.numpy(), feats.numpy(), opac.numpy(), tile=8)
    assert int(state.n_visible) == len(st.sorted_points) and int(state.n_instances) == len(st.inst_point)
    dbg = R.debug_arrays(state, settings, blobs.point, blobs.instance)
    assert np.array_equal(dbg["sorted_points"].cpu().numpy().view(np.uint32), st.sorted_points)
    assert np.array_equal(dbg["inst_point"].cpu().numpy().view(np.uint32), st.inst_point)
    assert np.array_equal(dbg["ranges"].cpu().numpy().view(np.uint32), st.ranges)
    assert np.array_equal(dbg["bounds"].cpu().numpy().view(np.uint16), st.bounds)
    return int(state.n_visible)


# blocks of 256 points, histogram blocks of 16384, tiles of 2048 pairs up to 2^18 points, of 8192 above
@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 2047, 2048, 2049, 16385, (1 << 18) - 1, (1 << 18) + 1, 8192 * 33 + 5])
@pytest.mark.parametrize("pattern", ["all", "none", "half", "one", "rows", "front", "back"])
def test_points_that_are_culled_keep_out_of_the_order(n, pattern):
    i = torch.arange(n)
    seen = {"all": i >= 0, "none": i < 0, "half": torch.rand(n, generator=torch.Generator().manual_seed(n)) < 0.5, "one": i == n // 2,
            "rows": (i // 32) % 3 == 1, "front": i < n // 3, "back": i >= n - n // 3}[pattern]
    visible = _check(*_scene(n, seen, n))
    assert visible <= int(seen.sum())


# Planes whose key range is 27 bits, exactly 30 bits of ones (a splat of four tiles at the far plane must not look culled), 31 bits, and 32 for a near plane
# that is not positive
@pytest.mark.parametrize("near, far", [(0.01, 100.0), (1.0, float(np.finfo(np.float32).max)), (0.5, float(np.finfo(np.float32).max)), (0.0, 100.0)])
def test_key_ranges_next_to_the_mark_of_a_culled_point(near, far):
    n = 5000
    view, pos, opac = _scene(n, torch.arange(n) % 3 != 0, 7, near, far)
    assert _check(view, pos, opac) > n // 2


# No depth is behind a far plane that is no number: the keys have to hold all of them, as with a plane at infinity
@pytest.mark.parametrize("near", [0.01, 0.0])
def test_a_far_plane_that_is_no_number(near):
    import inpc_b200
    from inpc_b200.views import look_at_view
    n = 4000
    g = torch.Generator().manual_seed(11)
    pos = torch.rand((n, 3), generator=g) * 2 - 1
    pos = (torch.tensor([0.0, 0.0, 3.0]) + (pos - torch.tensor([0.0, 0.0, 3.0])) * torch.exp(torch.rand((n, 1), generator=g) * 40)).contiguous().to(DEV)
    feats, rows = torch.randn((n, 36), generator=g).to(torch.float16).to(DEV), torch.randn((n, 8), generator=g).to(DEV)
    opac = (torch.rand((n, 1), generator=g) * 0.2).to(DEV)
    out = []
    for far in (float("inf"), float("nan")):
        view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 72, 40, 64.0, 64.0, near_plane=near, far_plane=far).to(DEV)
        rast = {tile: inpc_b200.INPCRasterizer(tile_size=tile) for tile in (8, 16)}
        out.append([rast[tile](view, mode, pos, feats, opac) for tile in (8, 16) for mode in (0, 1)] + [rast[tile].forward_rows(view, pos, rows, opac) for tile in (8, 16)])
    assert float(out[0][0][1].max()) > 0.3
    for a, b in zip(*out):
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
        # sums of atomic additions in any order
        assert float((a[2] - b[2]).abs().max()) <= 32 * 2.0 ** -24 * float(a[2].max())


# Splats that lie exactly between two pixels, also at the edges of tiles (no second tile is touched) and at the border of the image, in front of it and behind it,
# beside others: their footprints do not follow from the codes that the depth sort carries along.  One tile; a few; so many that the codes do not fit beside
# 32-bit keys (near plane at zero), where the words are gathered instead, as where keys are sorted in one pass (planes close together); both sizes of the sort's tiles.
@pytest.mark.parametrize("width, height", [(8, 8), (64, 24), (1024, 1040)])
@pytest.mark.parametrize("near, far", [(0.01, 100.0), (0.0, 100.0), (1.0, 1.0 + 2.0 ** -16)])
@pytest.mark.parametrize("n", [3000, (1 << 18) + 77])
def test_footprints_that_end_exactly_at_a_tile(width, height, near, far, n):
    from inpc_b200.views import look_at_view
    g = torch.Generator().manual_seed(n + width)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, height, float(width), float(width), near_plane=near, far_plane=far)
    depth = torch.tensor([1.0, 2.0, 4.0])[torch.randint(0, 3, (n,), generator=g)]
    px, py = ((torch.randint(-2, 2 * s + 3, (n,), generator=g)) * 0.5 for s in (width, height))
    other = torch.rand(n, generator=g) < 0.5
    px, py = torch.where(other, px + torch.rand(n, generator=g) - 0.5, px), torch.where(other, py + torch.rand(n, generator=g) - 0.5, py)
    pos = torch.stack([(px - width / 2) / width * depth, -(py - height / 2) / width * depth, 3.0 - depth], dim=1).contiguous()
    assert _check(view, pos, torch.full((n, 1), 0.01)) > n // (5 if far < 2.0 else 2)


def test_codes_of_stacked_images():
    import inpc_b200
    from inpc_b200.views import look_at_view
    g = torch.Generator().manual_seed(5)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), 72, 40, 64.0, 64.0).to(DEV)
    sets = []
    for n in (5000, 1, 4097):
        px, py = torch.randint(-2, 147, (n,), generator=g) * 0.5, torch.randint(-2, 83, (n,), generator=g) * 0.5
        depth = torch.tensor([1.0, 2.0, 4.0])[torch.randint(0, 3, (n,), generator=g)]
        pos = torch.stack([(px - 36) / 64 * depth, -(py - 20) / 64 * depth, 3.0 - depth], dim=1).contiguous().to(DEV)
        sets.append((pos, (torch.randn((n, 37), generator=g) - 2.0).to(torch.float16).to(DEV)))
    images, depths, alphas = inpc_b200.INPCRasterizer(tile_size=8).render_multi(view, sets)
    for k, (pos, raw) in enumerate(sets):
        for tile in (8, 16):   # 16x16 tiles know no codes; sums in another order
            image, depth, alpha = inpc_b200.INPCRasterizer(tile_size=tile).render(view, 0, pos, raw, 1.0, 3.0)
            for a, b in ((images[k], image), (depths[k], depth), (alphas[k], alpha)):
                assert torch.equal(a, b) if tile == 8 else torch.allclose(a, b, rtol=1e-5, atol=1e-5)
        assert k == 1 or float(alpha.max()) > 0.1
