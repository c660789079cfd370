"""Kernels at the sizes where a tile, a remainder or a dispatch rule can go wrong, against the same sums in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
U = 2.0 ** -24   # unit roundoff of float32


def _linear64(W, x, inds):
    r = x.double().reshape(x.shape[0], x.shape[1], -1)
    return torch.einsum("oi,ris->ros", W.double(), r).reshape(x.shape[0], W.shape[0], *x.shape[2:])


# rows that leave ragged tiles on both sides of the small-tile rule (a tile holds 16 to 512 rows, 148 blocks), widths around
# the 32 / 64 / 128 outputs of a tile and the 8 / 16 channels of a step
@pytest.mark.parametrize("inds", [0, 1, 2])
@pytest.mark.parametrize("rows,dim_in,dim_out", [(1, 1, 1), (15, 7, 33), (513, 17, 32), (3001, 24, 65), (2500, 9, 129), (20003, 8, 31),
                                                 (9500, 40, 64)])
def test_tensor_linear_tiles(inds, rows, dim_in, dim_out):
    from ld_b200 import ops
    g = torch.Generator().manual_seed(rows + inds)
    W = torch.randn(dim_out, dim_in, generator=g)
    x = torch.randn(rows, dim_in, *[3] * inds, generator=g)
    dy = torch.randn(rows, dim_out, *[3] * inds, generator=g)
    y = ops.tensor_linear_fwd(inds, W.cuda(), x.cuda()).cpu().double()
    # a sum of n products in any order, with FMAs: |error| <= n u sum |w||x|
    bound = dim_in * U * _linear64(W.abs(), x.abs(), inds)
    assert bool(((y - _linear64(W, x, inds)).abs() <= bound).all())
    yt = ops.tensor_linear_fwd(inds, W.cuda().t(), dy.cuda()).cpu().double()   # strided weights
    assert bool(((yt - _linear64(W.t(), dy, inds)).abs() <= dim_out * U * _linear64(W.t().abs(), dy.abs(), inds)).all())
    dW = ops.tensor_linear_dw(inds, dy.cuda(), x.cuda(), dim_out, dim_in).cpu().double()
    flat = lambda t: t.double().reshape(rows, t.shape[1], -1)  # noqa: E731
    want = torch.einsum("ros,ris->oi", flat(dy), flat(x))
    size = torch.einsum("ros,ris->oi", flat(dy).abs(), flat(x).abs())
    assert bool(((dW - want).abs() <= rows * 3 ** inds * U * size).all())


@pytest.mark.parametrize("rows,chan", [(1, 1), (5, 7), (3, 32), (41, 33), (9000, 136)])   # warps with missing lanes, grid strides
def test_bee_products_tails(rows, chan):
    from ld_b200 import ops
    from oracle import reference_math as R
    g = torch.Generator().manual_seed(rows)
    t = [torch.randn(rows, chan, *[3] * (k % 3), generator=g) for k in range(6)]
    got = ops.bee_fwd(*[a.cuda() for a in t])
    want = R.bee(*[a.double() for a in t])
    size = R.bee(*[a.double().abs() for a in t])
    for k, (a, b, m) in enumerate(zip(got, want, size)):
        if k in (11, 12):   # cross products: both terms count with their size
            m = b.abs() + 2 * (t[1] if k == 11 else t[2]).double().abs().amax(-1, keepdim=True) * t[4].double().abs().amax(-1).reshape(
                rows, chan, *[1] * (k - 10))
        assert bool(((a.cpu().double() - b).abs() <= 10 * U * m).all()), k
