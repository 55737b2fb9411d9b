"""Sums of partial gradients over rows: the kernels for up to 8 rows of many columns, for few and for many rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [100, 65536, 65537, 70004])
@pytest.mark.parametrize("rows", [1, 3, 8, 9, 63, 64, 130])
def test_sum_over_rows(rows, n):
    import rwkv_cuda_b200 as R
    g = torch.Generator().manual_seed(rows + n)
    x = torch.randn(rows, n, generator=g)
    out = torch.full((n,), float("nan"), device="cuda")
    R.ops.reduce_batch_partials(x.cuda(), out)
    out = out.cpu()
    if rows <= 8:   # one row after the other
        want = torch.zeros(n)
        for r in x:
            want = want + r
        assert torch.equal(out, want)
    # each of at most `rows` additions rounds once, relative to partial sums below the sum of the sizes
    err = (out.double() - x.double().sum(0)).abs()
    assert (err <= rows * 2.0 ** -24 * x.double().abs().sum(0)).all()
