"""Norm backward for rows of more than 1024 columns (one pass, a block per row) and GELU in the product epilogues."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rms", [True, False])
@pytest.mark.parametrize("rows,C", [(1, 1032), (3, 2048), (700, 2048), (37, 2056), (5, 3072), (301, 3080), (150, 4096), (6, 4104), (9, 1100),
                                    (700, 1280), (445, 1288), (901, 1536), (30, 1544)])
def test_norm_backward_wide(rms, rows, C):
    """Around the widths where the block size changes; 4104 and 1100 columns take the row-per-warp kernels."""
    from incin_b200.ops import kernels as K
    g = torch.Generator().manual_seed(rows + C)
    x, dy, add = ((torch.randn(rows, C, generator=g) + o).to(torch.bfloat16).cuda() for o in (0.5, 0.0, 0.0))
    gamma = (torch.randn(C, generator=g) * 0.3 + 1).to(torch.bfloat16).cuda()
    xd, gd = x.double().requires_grad_(), gamma.double().requires_grad_()
    bd = torch.zeros(C, device="cuda").double().requires_grad_()
    if rms:
        rstd = (xd.detach().pow(2).mean(1) + 1e-5).rsqrt()
        y = xd * (xd.pow(2).mean(1, keepdim=True) + 1e-5).rsqrt() * gd
    else:
        mean = xd.detach().mean(1)
        rstd = (xd.detach().var(1, unbiased=False) + 1e-5).rsqrt()
        y = torch.nn.functional.layer_norm(xd, (C,), gd, bd, 1e-5)
    refs = torch.autograd.grad(y, (xd, gd) if rms else (xd, gd, bd), dy.double())
    dg, db = (torch.ones(C, device="cuda") for _ in range(2))      # accumulated into
    for fork in (add, None):
        dg.fill_(1.0), db.fill_(1.0)
        if rms:
            dx = K.rmsnorm_bwd(dy, x, gamma, rstd.float(), fork, dg)
        else:
            dx = K.layernorm_bwd(dy, x, gamma, mean.float(), rstd.float(), fork, dg, db)
        ref = refs[0] + (0 if fork is None else fork.double())
        # one rounding to bf16; the fp32 terms that add up to it are a few units large
        assert ((dx.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()
        assert ((dg.double() - 1 - refs[1]).abs() <= 1e-5 * rows ** 0.5 + 2e-6 * refs[1].abs()).all()
        if not rms:
            assert ((db.double() - 1 - refs[2]).abs() <= 1e-5 * rows ** 0.5 + 2e-6 * refs[2].abs()).all()


def _identity(n, k):
    eye = torch.zeros(n, k, dtype=torch.bfloat16, device="cuda")
    eye[:, :n] = torch.eye(n, device="cuda")
    return eye


@pytest.mark.parametrize("M,N", [(130, 264), (128, 44)])
def test_gelu_epilogues(M, N):
    """A product with the identity makes the epilogue's input known to the bit: [-14, 14] finely, tiny and huge values."""
    from incin_b200 import _native as nat
    from incin_b200.ops import gemm as G
    vals = torch.cat([torch.linspace(-14, 14, M * N - 8), torch.tensor([0.0, -0.0, 1e-30, -1e-30, 60.0, -60.0, 1e30, -1e30])])
    x = vals.view(M, N).to(torch.bfloat16).cuda()
    # diagonal product: x @ I over K = N
    K = (N + 7) // 8 * 8
    a = torch.zeros(M, K, dtype=torch.bfloat16, device="cuda")
    a[:, :N] = x
    eye = _identity(N, K)
    y, pre = torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    G.gemm(a, eye, y, M=M, N=N, K=K, lda=K, ldb=K, ldc=N, act=nat.ACT_GELU, aux=pre)
    assert torch.equal(pre, x)
    xd = x.double()
    cdf = 0.5 * torch.special.erfc(-xd * 0.5 ** 0.5)
    # the polynomial's relative error is 1.8e-6 down to x = -3 and 1.6e-3 at -12, a little more at -14; one rounding to bf16;
    # below 2^-126 the exponential is flushed to zero, 14 times which is 1.7e-37
    poly = torch.where(xd < -3, 2e-3, 4e-6)
    ref = xd * cdf
    assert ((y.double() - ref).abs() <= (2.0 ** -8 + poly) * ref.abs() + 2e-37).all()
    ones = torch.zeros(M, K, dtype=torch.bfloat16, device="cuda")
    ones[:, :N] = 1.0
    G.gemm(ones, eye, y, M=M, N=N, K=K, lda=K, ldb=K, ldc=N, act=nat.ACT_DGELU, aux=x)
    slope = torch.where(xd.abs() > 50, 0.0, xd * torch.exp(-0.5 * xd * xd) * 0.3989422804014327)
    ref = cdf + slope
    # (the two terms cancel near x = -0.75: each carries its own error)
    assert ((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + poly * (cdf + slope.abs()) + 2e-37).all()


def test_gelu_epilogues_nonfinite():
    """Infinities and NaN in either lane of a pair; their neighbours are as without them."""
    from incin_b200 import _native as nat
    from incin_b200.ops import gemm as G
    from incin_b200.ops import kernels as KN
    inf, nan = float("inf"), float("nan")
    M, N = 130, 96
    g = torch.Generator().manual_seed(1)
    plain = torch.randn(M, N, generator=g).to(torch.bfloat16).cuda()
    odd = plain.clone()
    spots = [(0, 0, inf), (1, 1, inf), (2, 34, -inf), (3, 95, -inf), (129, 64, nan), (128, 31, nan), (64, 7, inf), (64, 8, nan)]
    for r, c, v in spots:
        odd[r, c] = v
    hit = odd != plain
    # data gradient: the pre-activation comes from memory and is not mixed; at infinity its second term is infinity times zero
    ones, eye = torch.ones(M, N, dtype=torch.bfloat16, device="cuda"), _identity(N, N)
    got = []
    for pre in (plain, odd):
        y = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
        G.gemm(ones, eye, y, M=M, N=N, K=N, lda=N, ldb=N, ldc=N, act=nat.ACT_DGELU, aux=pre)
        got.append(y)
    assert torch.equal(got[0][~hit], got[1][~hit]) and torch.isnan(got[1][hit]).all()
    # forward: through the bias, column by column
    bias = torch.zeros(N, dtype=torch.bfloat16, device="cuda")
    G.gemm(plain, eye, got[0], M=M, N=N, K=N, lda=N, ldb=N, ldc=N, bias=bias, act=nat.ACT_GELU, aux=got[1])
    ref = got[0].clone()
    bias[[0, 35, 64]] = torch.tensor([inf, -inf, nan], dtype=torch.bfloat16, device="cuda")
    G.gemm(plain, eye, got[0], M=M, N=N, K=N, lda=N, ldb=N, ldc=N, bias=bias, act=nat.ACT_GELU, aux=got[1])
    assert (got[0][:, 0] == inf).all() and torch.isnan(got[0][:, [35, 64]]).all()   # gelu(-inf) is -inf times zero
    keep = torch.ones(N, dtype=torch.bool, device="cuda")
    keep[[0, 35, 64]] = False
    assert torch.equal(got[0][:, keep], ref[:, keep])
    out = KN.act_fwd(torch.tensor([inf, nan, 3.0], dtype=torch.bfloat16, device="cuda"), nat.ACT_GELU)
    assert out[0] == inf and torch.isnan(out[1]) and out[2] > 2.9
