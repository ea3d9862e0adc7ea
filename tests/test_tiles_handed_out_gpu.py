"""The tiles of the fused forward kernel: more of them than its CTAs can hold at a time (every accumulator set, tile
slot and residual slot is used again), tiles without any offset between full ones, a last sub-tile that is ragged or
missing, and two layers that run at once.  Small whole numbers: exact in any order."""
import pytest
import torch

from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SMS = 148


def _layer(tiles, c_in, c_out, seed):
    """A map of whole and ragged 128-row tiles with all, some or none of four offsets, and its operands."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    n = tiles * 128 - 77
    row = torch.arange(n, device=DEV)
    kind = torch.randint(0, 6, (tiles,), generator=gen, device=DEV)[row // 128]      # 0: no offset
    has = [(kind == 1) | (kind == 5), (kind == 2) | (kind == 5), (kind == 3) & (row % 3 == 0) | (kind == 5), (kind == 5) & (row % 2 == 0)]
    masks = torch.full((4, n), -1, dtype=torch.int32, device=DEV)
    for p, h in enumerate(has):
        masks[p, h] = torch.arange(int(h.sum()), dtype=torch.int32, device=DEV)
    sizes = (masks >= 0).sum(1).int()
    x = torch.randint(-2, 3, (n, c_in), generator=gen, device=DEV).half()
    w = torch.randint(-1, 2, (4, c_in, c_out), generator=gen, device=DEV).half()
    skip = torch.randint(-8, 9, (n, c_out), generator=gen, device=DEV).half()
    order = torch.arange(4, dtype=torch.int32, device=DEV)
    want = torch.zeros(n, c_out, device=DEV)
    for p, h in enumerate(has):
        want[h] += x[h].float() @ w[p].float()
    assert float(want.abs().max()) < 2000
    return (x, w, masks, masks.clone(), order, sizes), skip, want


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("sub_tiles", [1, 2])
@pytest.mark.parametrize("c_in,c_out", [(8, 32), (16, 40), (72, 48), (16, 64), (16, 128), (136, 96), (8, 256)])
@pytest.mark.parametrize("per_cta", [0.5, 5.3])
def test_tiles_of_one_layer(c_in, c_out, sub_tiles, residual, per_cta):
    tiles = int(per_cta * 2 * SMS) * sub_tiles + 1       # two CTAs an SM at most; an odd number of sub-tiles
    operands, skip, want = _layer(tiles, c_in, c_out, c_in + c_out)
    got = F.sparse_convolution_forward_fused(*operands, residual=skip if residual else None, algorithm="implicit",
                                             sub_tiles=sub_tiles)
    assert torch.equal(got.float(), want + skip.float() if residual else want)


@pytest.mark.parametrize("c_in,c_out", [(24, 64), (72, 64), (72, 20), (64, 256)])
@pytest.mark.parametrize("rows", [100, 128, 18_945, 37_888, 37_889, 75_777, 303_104, 303_105, 600_001])
def test_tiles_of_a_dense_layer(rows, c_in, c_out):
    """1x1x1 layers: dealt out or handed out, by their tiles and widths."""
    gen = torch.Generator(device=DEV).manual_seed(rows)
    x = torch.randint(-2, 3, (rows, c_in), generator=gen, device=DEV).half()
    w = torch.randint(-1, 2, (c_in, c_out), generator=gen, device=DEV).half()
    skip = torch.randint(-8, 9, (rows, c_out), generator=gen, device=DEV).half()
    want = x.float() @ w.float()
    assert torch.equal(F.dense_forward(x, w).float(), want)
    assert torch.equal(F.dense_forward(x, w, residual=skip).float(), want + skip.float())


def test_two_layers_at_once():
    """Blocks of one layer wait for places that the other one's hold, and both hand out their tiles."""
    layers = [_layer(2600, 16, 64, 1), _layer(2300, 136, 128, 2), _layer(1200, 8, 256, 3)]
    streams = [torch.cuda.Stream() for _ in layers]
    torch.cuda.synchronize()
    for _ in range(20):
        got = []
        for stream, (operands, skip, _) in zip(streams, layers):
            with torch.cuda.stream(stream):
                got.append(F.sparse_convolution_forward_fused(*operands, residual=skip, algorithm="implicit", sub_tiles=1))
        torch.cuda.synchronize()
        for out, (_, skip, want) in zip(got, layers):
            assert torch.equal(out.float(), want + skip.float())
