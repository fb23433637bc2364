"""GPU tests of kernels that count the digits of the keys they make for the sort behind them, and of the cloud whose bounding box is collected while it is
placed: at the edges of their blocks, bit for bit against the forms that do neither."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# groups of 1024 points, blocks that take several of them; images of one tile (nothing to sort by), of 2^7 tiles and one more, of more than 2^14; 2^18 tiles for three passes
@pytest.mark.parametrize("tile, width, height", [(8, 8, 8), (8, 16, 8), (8, 128, 64), (8, 136, 64), (8, 1032, 1024), (8, 4096, 4104), (16, 40, 24), (16, 2064, 2048)])
@pytest.mark.parametrize("n", [1, 1023, 1025, 400_001])
@pytest.mark.parametrize("mode", [0, 1])
def test_lists_of_points_counted_while_their_instances_are_emitted(tile, width, height, n, mode):
    from helpers import oracle_camera
    from inpc_b200 import rasterization as R
    from inpc_b200.views import look_at_view
    if n > 2000 and width * height > 1 << 21:
        pytest.skip("the oracle takes long")
    g = torch.Generator().manual_seed(n + width)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, height, float(width), float(width))
    z = torch.rand(n, generator=g)
    px, py = torch.rand(n, generator=g) * (width + 8) - 4, torch.rand(n, generator=g) * (height + 8) - 4
    pos = torch.stack([(px - width / 2) / width * (3 - z), -(py - height / 2) / width * (3 - z), z], dim=1).contiguous()
    feats, opac = torch.zeros((n, 36), dtype=torch.float16), torch.full((n, 1), 0.01)
    v = view.to(DEV)
    settings = R.INPCRasterizer.extract_settings(v, mode)
    _, _, _, state, blobs, _ = R.forward_with_state(pos.to(DEV), feats.to(DEV), opac.to(DEV), settings, tile)
    st = O.preprocess_and_order(mode, O.TRAIN, oracle_camera(view), pos.numpy(), feats.numpy(), opac.numpy(), tile=tile)
    dbg = R.debug_arrays(state, settings, blobs.point, blobs.instance)
    assert int(state.n_visible) == len(st.sorted_points) and int(state.n_instances) == len(st.inst_point)
    assert np.array_equal(dbg["inst_point"].cpu().numpy().view(np.uint32), st.inst_point)
    assert np.array_equal(dbg["ranges"].cpu().numpy().view(np.uint32), st.ranges)


@pytest.mark.parametrize("total", [1, 2, 31, 2047, 4097, 300_001])
@pytest.mark.parametrize("odd", [None, "negative", "zero", "nan", "infinite"])
def test_cloud_placed_with_its_box_is_the_cloud_ordered_afterwards(total, odd):
    from inpc_b200 import sampling as S
    g = torch.Generator().manual_seed(total)
    leaves = 700
    centers = torch.rand((leaves, 3), generator=g) * 2 - 1
    levels = torch.randint(2, 9, (leaves,), generator=g, dtype=torch.int32)
    weights = torch.rand(leaves, generator=g)
    if odd == "negative":
        centers = centers - 5.0
    elif odd == "zero":
        centers[:, 1] = -0.0
    elif odd is not None:
        centers[leaves // 2, 2] = float("nan") if odd == "nan" else float("inf")
    c, l, w = centers.to(DEV), levels.to(DEV), weights.to(DEV)
    cloud = S.extract_global(S.ProbabilityFieldSampler(3), c, l, w, [], total, 2.0)
    plain = S.extract_global(S.ProbabilityFieldSampler(3), c, l, w, [], total, 2.0, use_morton_order=False)
    assert torch.equal(cloud.view(torch.int32), S.morton_order(plain).view(torch.int32))


# The counts a forward leaves on the device are three, made independently (points in the depth sort, instances by its keys, instances
# emitted): one that contradicts the others is an error.  Images of many tiles, and of one, whose instances the emission does not count.
@pytest.mark.parametrize("width, height", [(40, 24), (8, 8)])
@pytest.mark.parametrize("word, change", [(0, 10_000), (0, -(1 << 40)), (1, -1), (1, 1 << 20), (2, -1), (2, 1)])
def test_counts_that_contradict_one_another(width, height, word, change):
    from inpc_b200 import _cabi
    from inpc_b200 import rasterization as R
    from inpc_b200.views import look_at_view
    n = 5000
    g = torch.Generator().manual_seed(word)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, height, 40.0, 40.0).to(DEV)
    pos, opac = (torch.rand((n, 3), generator=g) * 2 - 1).to(DEV), torch.full((n, 1), 0.01, device=DEV)
    settings = R.INPCRasterizer.extract_settings(view, 0)
    _, _, _, state, blobs, _ = R.forward_with_state(pos, torch.zeros((n, 36), dtype=torch.float16, device=DEV), opac, settings, 8)
    want = (state.n_visible, state.n_instances)
    words = blobs.point[:blobs.point.numel() // 8 * 8].view(torch.int64)
    at = torch.nonzero((words[:-2] == want[0]) & (words[1:-1] == want[1]) & (words[2:] == want[1])).reshape(-1)
    assert at.numel() == 1 and 0 < want[0] < n
    R.resolve_counts(state)
    assert (state.n_visible, state.n_instances) == want
    words[at[0] + word] += change
    with pytest.raises(_cabi.InpcError, match="inconsistent counts"):
        R.resolve_counts(state)
    words[at[0] + word] -= change
    R.resolve_counts(state)
    assert (state.n_visible, state.n_instances) == want


# Runs of the tile keys that end at, before and behind the first key of a thread (every 16th) and of a warp (every 512th), behind the last whole group of either, and empty tiles
@pytest.mark.parametrize("lengths", [(1,), (16,), (16, 16, 480), (15, 1, 16, 17, 463, 1, 511, 0, 0, 513), (512, 512, 511), (0, 1024, 1, 0), (1000, 0, 40, 7, 17, 16), (0, 2048, 2048, 15)])
@pytest.mark.parametrize("tile", [8, 16])
def test_ranges_of_runs_that_end_beside_a_threads_keys(lengths, tile):
    from inpc_b200 import rasterization as R
    from inpc_b200.views import look_at_view
    width = tile * len(lengths)
    view = look_at_view((0.0, 0.0, 3.0), (0.0, 0.0, 0.0), width, tile, float(width), float(width)).to(DEV)
    n = sum(lengths)
    px = torch.repeat_interleave(torch.arange(len(lengths)) * tile + tile / 2, torch.tensor(lengths))
    z = torch.rand(n, generator=torch.Generator().manual_seed(n))
    pos = torch.stack([(px - width / 2) / width * (3 - z), torch.zeros(n), z], dim=1)[torch.randperm(n, generator=torch.Generator().manual_seed(1))].contiguous()
    settings = R.INPCRasterizer.extract_settings(view, 0)
    _, _, _, state, blobs, _ = R.forward_with_state(pos.to(DEV), torch.zeros((n, 36), dtype=torch.float16, device=DEV), torch.full((n, 1), 0.01, device=DEV), settings, tile)
    ranges = R.debug_arrays(state, settings, blobs.point, blobs.instance)["ranges"].cpu()
    ends = np.cumsum(lengths)
    assert ranges.tolist() == [[int(e) - k, int(e)] if k else [0, 0] for e, k in zip(ends, lengths)]
