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
