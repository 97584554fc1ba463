"""Surrogate kernels at the ends of their index ranges."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2**31 - 1, 2**31 - 512])
def test_colsum_of_the_most_rows(product, rows):
    """One column of (nearly) 2^31 rows: the row index steps past 2^31 after the last row.  Zeros with
    ones in the last thousand rows, so the sum is exact and a lost tail shows."""
    import torch
    from soltrace_b200.surrogate import Mlp
    net = Mlp(product, dims=(16, 256, 256), seed=1)
    dz = torch.zeros(rows, 1, dtype=torch.bfloat16, device="cuda")
    dz[-1000:] = 1.0
    db = torch.full((1,), 7.0, device="cuda")
    fn = product.lib.st_b200_mlp_colsum
    assert fn(rows, 1, dz.data_ptr(), db.data_ptr(), net._s()) == 1
    torch.cuda.synchronize()
    assert db.item() == 1000.0
