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


@pytest.mark.parametrize("rows", [64, 100, 256])
def test_errors_of_a_sum_over_many_rows(rows):
    """Against fp64 no larger than with eight strands added one after the other (the form for fewer rows); 2 % for the sample of 70004 sums."""
    import rwkv_cuda_b200 as R
    x = torch.randn(rows, 70004, generator=torch.Generator().manual_seed(rows))
    out = torch.empty(70004, device="cuda")
    R.ops.reduce_batch_partials(x.cuda(), out)
    strands = torch.zeros(8, 70004)
    for i, r in enumerate(x):
        strands[i % 8] += r
    eight = strands[0].clone()
    for s in strands[1:]:
        eight += s
    want = x.double().sum(0)
    assert (out.cpu().double() - want).norm() <= 1.02 * (eight.double() - want).norm()
