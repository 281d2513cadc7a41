"""Tiled convolution helpers, cluster batch norm and pooling at the sizes where their tiles end."""
import pytest
import torch
import torch.nn.functional as TF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N,C,H,W,k,s,p,d", [
    (2, 8, 9, 9, (3, 3), (1, 1), (1, 1), (1, 1)),         # one channel tile, a band of one row at the end
    (1, 24, 17, 5, (3, 3), (2, 2), (1, 1), (1, 1)),       # the last channel tile is half empty
    (3, 72, 8, 33, (1, 1), (1, 1), (0, 0), (1, 1)),
    (2, 16, 12, 40, (5, 3), (2, 1), (2, 0), (1, 2)),
    (1, 8, 5, 700, (3, 3), (1, 1), (1, 1), (1, 1)),       # a line longer than a block's tile can be in bands of eight
    (1, 8, 4, 3000, (3, 3), (1, 1), (1, 1), (1, 1)),      # does not fit at all: general kernels
    (2, 3, 10, 10, (3, 3), (1, 1), (1, 1), (1, 1)),       # K = 27: general kernels
    (2, 4, 6, 6, (2, 2), (3, 3), (0, 0), (1, 1)),         # pixels that no window reads
    # large enough for the tiled kernels: odd lines, a half empty channel tile, dilation, one-row bands, strides, 1 x 1
    (16, 64, 17, 33, (3, 3), (1, 1), (1, 1), (1, 1)),
    (40, 24, 20, 21, (3, 3), (1, 1), (1, 1), (1, 1)),
    (12, 40, 30, 19, (3, 3), (1, 1), (2, 2), (2, 2)),
    (20, 16, 30, 90, (3, 3), (1, 1), (1, 1), (1, 1)),
    (8, 40, 41, 50, (5, 3), (2, 1), (2, 0), (1, 2)),
    (24, 72, 30, 31, (1, 1), (1, 1), (0, 0), (1, 1)),
    (9, 64, 19, 17, (4, 4), (1, 1), (3, 3), (1, 1)),
])
def test_im2col_col2im_tiles(dtype, N, C, H, W, k, s, p, d):
    from incin_b200.ops import tensor_ops as T
    g = torch.Generator().manual_seed(H * W)
    # whole numbers of few bits: every sum is exact in both types
    x = torch.randint(-4, 5, (N, C, H, W), generator=g).to(dtype).cuda()
    cols = T.im2col(x, k, s, p, d)
    ref = TF.unfold(x.float(), k, d, p, s).transpose(1, 2).reshape(cols.shape)
    assert torch.equal(cols.float(), ref)
    gcols = torch.randint(-2, 3, cols.shape, generator=g).to(dtype).cuda()
    L = cols.shape[0] // N
    back = TF.fold(gcols.float().reshape(N, L, -1).transpose(1, 2), (H, W), k, d, p, s)
    assert torch.equal(T.col2im(gcols, x.shape, k, s, p, d).float(), back)
    odd = torch.zeros(gcols.numel() + 1, dtype=dtype, device="cuda")      # a column matrix that is not 16-byte aligned
    odd[1:] = gcols.reshape(-1)
    assert torch.equal(T.col2im(odd[1:].view(gcols.shape), x.shape, k, s, p, d).float(), back)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(1, 1, 1, 2), (2, 3, 1, 1), (5, 7, 3, 3), (64, 2, 16, 16), (9, 5, 40, 8), (33, 600, 8, 8), (70, 64, 15, 31)])
def test_batch_norm_slices(dtype, shape):
    """One to eight CTAs a channel, with and without 16-byte accesses; a large mean; forward and backward in 64 bits."""
    from incin_b200.ops import tensor_ops as T
    g = torch.Generator().manual_seed(sum(shape))
    x = (torch.randn(shape, generator=g) + 5.0).to(dtype).cuda().requires_grad_()
    dy = torch.randn(shape, generator=g).to(dtype).cuda()
    ga, be = (torch.randn(shape[1], generator=g).cuda().requires_grad_() for _ in range(2))
    rm, rv = torch.zeros(shape[1], device="cuda"), torch.ones(shape[1], device="cuda")
    y = T.batch_norm(x, ga, be, rm, rv, True, 0.1, 1e-5)
    dx, dga, dbe = torch.autograd.grad(y, (x, ga, be), dy)
    xd, gd, bd = (t.detach().double().requires_grad_() for t in (x, ga, be))
    rmd, rvd = torch.zeros(shape[1], device="cuda").double(), torch.ones(shape[1], device="cuda").double()
    yd = TF.batch_norm(xd, rmd, rvd, gd, bd, True, 0.1, 1e-5)
    refs = torch.autograd.grad(yd, (xd, gd, bd), dy.double())
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -18     # one rounding of the output / fp32 sums and the variance's differences
    n = x.numel() // shape[1]
    for got, ref, scale in ((y, yd, 1.0), (dx, refs[0], 1.0), (dga, refs[1], n ** 0.5), (dbe, refs[2], n ** 0.5), (rm, rmd, 1.0), (rv, rvd, 1.0)):
        floor = (2.0 ** -14 * scale + 1e-5) * (1.0 + ref.abs().max())
        assert ((got.double() - ref).abs() <= u * ref.abs() + floor).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape,k,s,p", [((1, 1, 1, 1), 1, 1, 0), ((3, 5, 7, 33), 3, 2, 1), ((2, 9, 8, 8), 2, 2, 0), ((2, 3, 40, 65), (3, 2), (1, 3), (1, 0)),
                                         ((1, 2, 1, 70001), (1, 3), (1, 2), (0, 1)), ((2, 1, 30001, 1), (2, 1), (2, 1), (0, 0))])
def test_max_pool_shapes(dtype, shape, k, s, p):
    from incin_b200.ops import tensor_ops as T
    g = torch.Generator().manual_seed(shape[-1])
    x = torch.randn(shape, generator=g).to(dtype).cuda().requires_grad_()
    xr = x.detach().float().requires_grad_()
    y, yr = T.max_pool2d(x, k, s, p), TF.max_pool2d(xr, k, s, p)
    assert torch.equal(y.float(), yr)
    dy = torch.randint(-2, 3, y.shape, generator=g).to(dtype).cuda()
    assert torch.equal(torch.autograd.grad(y, x, dy)[0].float(), torch.autograd.grad(yr, xr, dy.float())[0])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("planes,hw,out", [((2, 3), (7, 5), (3, 2)), ((1, 4), (5, 7), (8, 9)), ((3, 1), (1, 50001), (1, 7)), ((2, 2), (40, 1), (6, 1)),
                                           ((2, 8), (16, 16), (4, 4)), ((1, 1), (1, 1), (1, 1)), ((1, 2), (1, 9), (1, 4000))])
def test_adaptive_pool_shapes(dtype, planes, hw, out):
    from incin_b200.ops import tensor_ops as T
    g = torch.Generator().manual_seed(hw[1])
    x = torch.randn(*planes, *hw, generator=g).to(dtype).cuda().requires_grad_()
    xd = x.detach().double().requires_grad_()
    y, yd = T.adaptive_avg_pool2d(x, out), TF.adaptive_avg_pool2d(xd, out)
    dy = torch.randn(y.shape, generator=g).to(dtype).cuda()
    dx, dxd = torch.autograd.grad(y, x, dy)[0], torch.autograd.grad(yd, xd, dy.double())[0]
    # fp32 sums of up to in / out or out / in terms, quotients of 2^-22 (--use_fast_math), one rounding to the type
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -21
    for got, ref in ((y, yd), (dx, dxd)):
        assert ((got.double() - ref).abs() <= u * ref.abs() + 2.0 ** -16 * ref.abs().max() + 1e-7).all()


@pytest.mark.parametrize("perm", [(0, 2, 3, 1), (0, 3, 1, 2), (1, 0, 2, 3), (3, 2, 1, 0)])
@pytest.mark.parametrize("shape", [(2, 3, 4, 5), (1, 8, 1, 16), (4, 64, 8, 9), (3, 1, 1, 7), (1, 1, 1, 1)])
def test_strided_copy_merged_axes(shape, perm):
    from incin_b200.ops import tensor_ops as T
    x = torch.arange(torch.tensor(shape).prod().item(), device="cuda", dtype=torch.float32).view(shape)
    for t in (x, x.bfloat16()):
        assert torch.equal(T.materialize(t.permute(perm)), t.permute(perm).contiguous())
    wide = x[:, :, :, None].expand(*shape[:3], 3, shape[3])
    assert torch.equal(T.materialize(wide), wide.contiguous())


def test_more_than_two_to_the_31_elements():
    """Flat indexes of 64 bits: windows and cells of one element, so that every result is a copy of its input."""
    from incin_b200.ops import tensor_ops as T
    shape = (1, 3, 26755, 26756)
    x = torch.empty(shape, dtype=torch.bfloat16, device="cuda").random_(-100, 100)
    assert x.numel() > 2 ** 31
    for op in (lambda t: T.max_pool2d(t, 1), lambda t: T.adaptive_avg_pool2d(t, shape[2:])):
        leaf = x.detach().requires_grad_()
        y = op(leaf)
        assert torch.equal(y, x)
        assert torch.equal(torch.autograd.grad(y, leaf, x)[0], x)
        del y, leaf
    cols = T.im2col(x, (1, 1))                  # K = 3: the general kernels
    assert torch.equal(cols.view(*shape[2:], 3), x[0].permute(1, 2, 0))
    assert torch.equal(T.col2im(cols, shape, (1, 1)), x)
