"""Sub-tiles of one CTA tile of the fused forward kernel that have no offset in common, or none at all:
what one sub-tile lacks is neither copied nor multiplied for it.  With and without a residual, which comes through
shared memory at 33 to 64 columns.  Small whole numbers: exact in any order."""
import pytest
import torch

from minuet_b200.nn import functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _masks(rows_of):
    """Masks and sizes of a map whose target t has source t under the offsets of ``rows_of[p]``."""
    n = int(max(int(r.max()) for r in rows_of if len(r))) + 300
    source = torch.full((len(rows_of), n), -1, dtype=torch.int32, device=DEV)
    for p, r in enumerate(rows_of):
        source[p, r] = torch.arange(len(r), dtype=torch.int32, device=DEV)
    return source, source.clone(), torch.tensor([len(r) for r in rows_of], dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("sub_tiles", [0, 1, 2])
@pytest.mark.parametrize("c_in,c_out", [(8, 16), (32, 32), (24, 40), (64, 48), (72, 64), (128, 128), (64, 256)])
def test_sub_tiles_without_offsets_in_common(c_in, c_out, sub_tiles):
    gen = torch.Generator(device=DEV).manual_seed(c_in + c_out)
    at = lambda first, count: torch.arange(first, first + count, device=DEV)
    # tiles (rows keep their order): offsets 0 | 1, none | 2, 0 and 2 | none, 1 | 1 and 3, a ragged end
    rows_of = [torch.cat([at(0, 128), at(512, 100)]), torch.cat([at(128, 128), at(768, 256)]),
               torch.cat([at(384, 128), at(540, 100)]), torch.cat([at(900, 124), at(1024, 33)])]
    sm, tm, sizes = _masks(rows_of)
    n = sm.shape[1]
    x = torch.randint(-2, 3, (n, c_in), generator=gen, device=DEV).half()
    w = torch.randint(-1, 2, (4, c_in, c_out), generator=gen, device=DEV).half()
    skip = torch.randint(-8, 9, (n, c_out), generator=gen, device=DEV).half()
    order = torch.tensor([2, 0, 3, 1], dtype=torch.int32, device=DEV)
    want = torch.zeros(n, c_out, device=DEV)
    for p, r in enumerate(rows_of):
        want[r] += x[r].float() @ w[order[p].long()].float()
    assert float(want.abs().max()) < 2000
    got = F.sparse_convolution_forward_fused(x, w, sm, tm, order, sizes, algorithm="implicit", sub_tiles=sub_tiles)
    assert torch.equal(got.float(), want)
    got = F.sparse_convolution_forward_fused(x, w, sm, tm, order, sizes, residual=skip, algorithm="implicit",
                                             sub_tiles=sub_tiles)
    assert torch.equal(got.float(), want + skip.float())
