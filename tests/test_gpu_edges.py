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
@pytest.mark.parametrize("total,gap", [(1, 0), (2047, 0), (2048, 1), (2049, 3000), (6145, 2049), (20_000, 2047)])
def test_halton_samples_over_runs_of_empty_leaves(total, gap):
    from inpc_b200.sampling import halton_samples
    g = torch.Generator().manual_seed(total)
    filled = torch.randint(1, 40, (max(1, total // 17),), generator=g)
    filled[-1] += max(0, total - int(filled.sum()))
    counts = torch.zeros(len(filled) * 2 + gap * 3, dtype=torch.int32)
    at = torch.arange(len(filled)) * 2
    at[len(filled) // 2:] += gap
    at[len(filled) * 3 // 4:] += gap
    counts[at] = filled.to(torch.int32)
    n = counts.numel()
    centers = torch.rand((n, 3), generator=g) * 2 - 1
    levels = torch.randint(0, 11, (n,), generator=g, dtype=torch.int32)
    out = halton_samples(counts.to(DEV), centers.to(DEV), levels.to(DEV), 2.0)
    np.testing.assert_array_equal(out.cpu().numpy(), O.halton_samples(counts.numpy(), centers.numpy(), levels.numpy(), 2.0))
