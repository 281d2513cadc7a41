"""SwiGLU and rotary embedding: the 16-byte kernels and the element-wise ones at the sizes between them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,F", [(1, 8), (3, 5), (7, 12), (33, 40), (5, 2816), (1000, 264)])
@pytest.mark.parametrize("shift", [0, 1])
def test_swiglu(rows, F, shift):
    """``shift``: bases that are not 16-byte aligned."""
    from incin_b200.ops import functional as FN
    g = torch.Generator().manual_seed(F)
    def mk(*shape):
        n = rows * shape[-1]
        flat = torch.zeros(n + shift, dtype=torch.bfloat16, device="cuda")
        flat[shift:] = torch.randn(n, generator=g).to(torch.bfloat16).cuda()
        return flat[shift:].view(shape)
    gu, dy = mk(rows, 2 * F).requires_grad_(), mk(rows, F)
    y = FN.swiglu(gu)
    (dgu,) = torch.autograd.grad(y, gu, dy)
    d = gu.detach().double().requires_grad_()
    yd = torch.nn.functional.silu(d[:, :F]) * d[:, F:]
    (dd,) = torch.autograd.grad(yd, d, dy.double())
    for got, ref in ((y, yd), (dgu, dd)):   # one rounding to bf16 (2^-8), fp32 before it
        assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-5).all()


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("B,T,H,D", [(1, 1, 1, 16), (2, 7, 3, 64), (3, 9, 4, 128), (1, 33, 2, 8), (2, 5, 2, 24), (1, 19, 36, 64), (2, 3, 1, 256),
                                     (1, 1, 126, 256), (1, 8, 125, 128), (3, 200, 3, 64), (1, 2500, 2, 32)])
def test_rope(B, T, H, D, inverse):
    """Rotation of the first H of H + 2 heads in place; D / 2 no multiple of 8 takes the element-wise kernel."""
    from incin_b200.ops import kernels as K
    g = torch.Generator().manual_seed(D + T)
    x = torch.randn(B, T, H + 2, D, generator=g).to(torch.bfloat16).cuda()
    ref = x.double().clone()
    half = D // 2
    ang = torch.arange(T).double()[:, None] * 10000.0 ** (-2.0 * torch.arange(half).double() / D)
    cs, sn = ang.cos().cuda()[None, :, None], ang.sin().cuda()[None, :, None] * (-1.0 if inverse else 1.0)
    a, c = ref[:, :, :H, :half].clone(), ref[:, :, :H, half:].clone()
    ref[:, :, :H, :half], ref[:, :, :H, half:] = a * cs - c * sn, c * cs + a * sn
    y = K.rope_out(x, H, 10000.0, inverse)
    assert torch.equal(y[:, :, H:], x[:, :, H:])
    K.rope_(x, B, T, H, D, T * (H + 2) * D, (H + 2) * D, D, 10000.0, inverse)
    # one rounding to bf16, and angles up to T in fp32 (2^-22 of the angle, hardware sine and cosine)
    assert ((x.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (T * 2.0 ** -20 + 1e-5) * 4).all()
    assert torch.equal(y, x)
