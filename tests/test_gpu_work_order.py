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
