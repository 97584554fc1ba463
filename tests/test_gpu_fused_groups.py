"""Group sums of the fused surrogate forward: the output layer's products run transposed there (a
thread owns an output and walks the tile's rows), so groups may begin and end at any row of a tile
or of the 32-row pieces it is read in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (8, 256, 256, 512)
CASES = [(rows, group) for rows in (1, 31, 129, 419, 40_001) for group in (1, 31, 32, 33, 128, 200, 50_000)]


@pytest.mark.parametrize("rows,group", CASES)
@pytest.mark.parametrize("clamp", (False, True))
def test_group_sums_match_rows(product, rows, group, clamp):
    """The sums equal those of the rows that the same kernel writes.  A row of either orientation
    agrees to 1e-5 of the largest (float accumulation of 256 terms); a sum adds at most five
    levels and four pieces of a tile and one atomic per tile, each rounding once."""
    import torch
    from soltrace_b200.surrogate import Mlp
    net = Mlp(product, dims=DIMS, seed=5)
    rng = np.random.default_rng(rows)
    for b in net.b:
        b.copy_(torch.from_numpy(rng.normal(scale=0.1, size=b.numel()).astype(np.float32)))
    x = torch.from_numpy(rng.normal(size=(rows, DIMS[0])).astype(np.float32)).to(torch.bfloat16).cuda()
    each = net.forward_fused(x, group_rows=0, scale=0.5, clamp=clamp).double()
    got = net.forward_fused(x, group_rows=group, scale=0.5, clamp=clamp).double()
    torch.cuda.synchronize()
    assert net.error() == 0
    index = torch.arange(rows, device="cuda") // group
    zero = torch.zeros(-(-rows // group), DIMS[-1], dtype=torch.float64, device="cuda")
    want, size = zero.index_add(0, index, each), zero.index_add(0, index, each.abs())
    assert got.shape == want.shape
    limit = (1e-5 + (10 + rows / 128) * 2.0**-24) * size.max().item()
    assert (got - want).abs().max().item() <= limit
