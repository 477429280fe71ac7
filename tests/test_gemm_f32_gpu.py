"""The float32 product at the ends of its tiles, aligned and not, added and stored; a row's bits do not depend on the rows beside it,
whichever tile the product is cut into."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,pad", [(1, 1, 1, 0), (31, 33, 15, 0), (33, 65, 17, 3), (64, 64, 16, 0), (65, 130, 36, 4), (200, 900, 100, 0),
                                       (640, 1000, 52, 1), (577, 1025, 33, 0)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_product_is_a_float32_sum(m, n, k, pad, accumulate):
    from celeg_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    x = torch.randn(m, k + pad, device="cuda", generator=g)[:, :k]
    w = torch.randn(n, k, device="cuda", generator=g)
    before = torch.randn(m, n, device="cuda", generator=g)
    y = before.clone()
    kernels.gemm_f32(x, w, y, m, accumulate=accumulate)
    want = x.double() @ w.double().T + (before.double() if accumulate else 0.0)
    # a sum of k products in order: k roundings of 2^-24 of the sum of the products' sizes at most
    bound = (k + 2) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + before.double().abs())
    assert bool(((y.double() - want).abs() <= bound).all())


def test_a_row_does_not_depend_on_the_rows_beside_it():
    from celeg_b200 import kernels
    g = torch.Generator(device="cuda").manual_seed(3)
    x, w = torch.randn(700, 260, device="cuda", generator=g), torch.randn(1100, 260, device="cuda", generator=g)
    many, few = torch.empty(700, 1100, device="cuda"), torch.empty(3, 1100, device="cuda")
    kernels.gemm_f32(x, w, many, 700)                     # tiles of 64 x 64
    kernels.gemm_f32(x[200:203], w, few, 3)               # of 32 x 32
    assert torch.equal(many[200:203], few)


def test_as_many_rows_as_a_launch_has_tiles_of_64():
    from celeg_b200 import kernels
    w = torch.full((1, 1), 3.0, device="cuda")
    for rows in (32 * 65535, 32 * 65535 + 1, 64 * 65535):
        x = torch.arange(rows, device="cuda").float()[:, None]
        y = torch.empty_like(x)
        kernels.gemm_f32(x, w, y, rows)
        assert torch.equal(y, x * 3.0)
    with pytest.raises(kernels.KernelLibraryError, match="exceed one launch"):
        kernels.gemm_f32(x, w, y, 64 * 65535 + 1)
