"""Attention kernels at the sizes where their pipelines change shape (first and last tiles, one tile per work item)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,H,D", [(8, 128, 32, 64), (6, 626, 32, 64), (8, 200, 24, 128)])
def test_backward_repeats_to_the_bit(B, T, H, D):
    """dK and dV have a fixed summation order, so repeated backward passes agree bit for bit; a product that starts
    before its operands are complete shows up as a difference (most likely in items of one query tile)."""
    from incin_b200.ops import attention as A
    from incin_b200.ops import gemm as G
    g = torch.Generator().manual_seed(3)
    q, k, v, do = (torch.randn(B, T, H, D, generator=g).to(torch.bfloat16).cuda() for _ in range(4))
    q, k, v = (t.requires_grad_() for t in (q, k, v))
    first = None
    for _ in range(24):
        out = A.flash_attention(q, k, v)
        _, dk, dv = torch.autograd.grad(out, (q, k, v), do)
        if first is None:
            first = (dk, dv)
        assert torch.equal(dk, first[0]) and torch.equal(dv, first[1])
    G.check_status()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,T,Hq,Hkv", [(1, 1, 1, 1), (2, 127, 3, 1), (1, 129, 2, 2), (3, 255, 2, 1), (1, 257, 4, 2),
                                        (40, 384, 6, 2), (2, 1025, 5, 5), (13, 128, 12, 4), (160, 64, 1, 1), (30, 192, 6, 6),
                                        (10, 300, 16, 2), (5, 640, 20, 20), (64, 65, 12, 12)])
def test_forward_tile_edges(B, T, Hq, Hkv, D):
    """Both kernels (one tile per CTA where pairs of tiles would leave SMs idle).  Query tiles come in pairs and items
    outnumber CTAs in some of these: one row, one tile, a pair with one tile beyond the sequence, several items per CTA;
    strided inputs; rows whose scores need rescaling on every tile."""
    from incin_b200.ops import attention as A
    from incin_b200.ops import gemm as G
    g = torch.Generator().manual_seed(T + D)
    x = torch.randn(B, T, Hq + 2 * Hkv, D, generator=g)
    # keys grow along the sequence so that the running maximum moves by more than the rescale threshold
    x[:, :, Hq:Hq + Hkv] *= torch.linspace(0.2, 6.0, T).view(1, T, 1, 1)
    x = x.to(torch.bfloat16).cuda()
    q, k, v = x[:, :, :Hq], x[:, :, Hq:Hq + Hkv], x[:, :, Hq + Hkv:]
    with torch.no_grad():
        out = A.flash_attention(q, k, v)
    G.check_status()
    s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double().repeat_interleave(Hq // Hkv, 2)) * D ** -0.5
    s = s.masked_fill(~torch.ones(T, T, device="cuda", dtype=torch.bool).tril(), float("-inf"))
    p, vd = torch.softmax(s, -1), v.double().repeat_interleave(Hq // Hkv, 2)
    ref = torch.einsum("bhqk,bkhd->bqhd", p, vd)
    # bf16 keeps 8 bits, so rounding P costs up to 2^-8 of each term and rounding the output 2^-8 more:
    # |error| <= 2^-8 (sum p |v| + |o|), 5 % above it for the fp32 scores, exponentials and sums
    bound = 2.0 ** -8 * 1.05 * (torch.einsum("bhqk,bkhd->bqhd", p, vd.abs()) + ref.abs()) + 1e-5
    assert ((out.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("B,T,Hq,Hkv,D", [(8, 1000, 12, 12, 64), (2, 2000, 32, 4, 64), (2, 2000, 24, 8, 128), (2, 1665, 32, 32, 128),
                                          (8, 300, 24, 8, 128), (13, 128, 12, 12, 64)])
def test_forward_repeats_to_the_bit(B, T, Hq, Hkv, D):
    """Every sum has a fixed order, so a product that starts before its operands are complete, or overwrites columns that
    another one still reads, shows up as a difference."""
    from incin_b200.ops import attention as A
    from incin_b200.ops import gemm as G
    g = torch.Generator().manual_seed(5)
    q, k, v = (torch.randn(B, T, h, D, generator=g).to(torch.bfloat16).cuda() for h in (Hq, Hkv, Hkv))
    with torch.no_grad():
        first = A.flash_attention(q, k, v)
        for _ in range(40):
            assert torch.equal(A.flash_attention(q, k, v), first)
    G.check_status()


@pytest.mark.parametrize("B,T,Hq,Hkv,D", [(2, 1665, 32, 32, 128), (2, 1665, 64, 64, 64), (3, 2300, 40, 20, 128)])
def test_forward_head_by_head(B, T, Hq, Hkv, D):
    """K and V of more than 48 MB: the items are walked head by head.  Several items per CTA, an odd number of tiles."""
    from incin_b200.ops import attention as A
    from incin_b200.ops import gemm as G
    assert B * Hkv * T * D * 4 > 48 << 20
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v = (torch.randn(B, T, h, D, generator=g, device="cuda").to(torch.bfloat16) for h in (Hq, Hkv, Hkv))
    with torch.no_grad():
        out = A.flash_attention(q, k, v)
    G.check_status()
    mask = torch.ones(T, T, device="cuda", dtype=torch.bool).tril()
    for b in range(B):
        for h in range(0, Hq, 8):
            heads = slice(h, h + 8)
            kv = torch.arange(h, h + 8, device="cuda") // (Hq // Hkv)
            qd, kd, vd = q[b, :, heads].double().transpose(0, 1), k[b, :, kv].double().transpose(0, 1), v[b, :, kv].double().transpose(0, 1)
            p = torch.softmax((qd @ kd.mT * D ** -0.5).masked_fill(~mask, float("-inf")), -1)
            ref = p @ vd
            bound = 2.0 ** -8 * 1.05 * (p @ vd.abs() + ref.abs()) + 1e-5   # as in test_forward_tile_edges
            assert ((out[b, :, heads].double().transpose(0, 1) - ref).abs() <= bound).all()


@pytest.mark.parametrize("B,T,Hq,Hkv", [(1, 900, 6, 2), (9, 384, 40, 40), (2, 1500, 16, 8)])
def test_backward_item_orders(B, T, Hq, Hkv):
    """head_dim 128 walks its work items longest first over all heads (few items) or head by head (1080 items here)."""
    from incin_b200.ops import attention as A
    from incin_b200.ops import gemm as G
    g = torch.Generator().manual_seed(T)
    q, k, v, do = (torch.randn(B, T, h, 128, generator=g).to(torch.bfloat16).cuda() for h in (Hq, Hkv, Hkv, Hq))
    leaves = [t.requires_grad_() for t in (q, k, v)]
    got = torch.autograd.grad(A.flash_attention(*leaves), leaves, do)
    G.check_status()
    grp, scale = Hq // Hkv, 128 ** -0.5
    qf, kf, vf, df = (t.detach().double().transpose(1, 2) for t in (q, k.repeat_interleave(grp, 2), v.repeat_interleave(grp, 2), do))
    mask = torch.ones(T, T, device="cuda", dtype=torch.bool).tril()
    for b in range(B):
        p = torch.softmax((qf[b] @ kf[b].mT * scale).masked_fill(~mask, float("-inf")), -1)
        o, dp = p @ vf[b], df[b] @ vf[b].mT
        delta = (df[b] * o).sum(-1, keepdim=True)
        ds = p * (dp - delta)
        # bf16 keeps 8 bits: P and dS are rounded before their products, O before delta = sum(dO O), the result at the end
        e = p * ((dp - delta).abs() + (df[b] * o).abs().sum(-1, keepdim=True))
        fold = lambda t: t.view(Hkv, grp, T, 128).sum(1)
        refs = (scale * ds @ kf[b], fold(scale * ds.mT @ qf[b]), fold(p.mT @ df[b]))
        slack = (scale * e @ kf[b].abs(), fold(scale * e.mT @ qf[b].abs()), fold(p.mT @ df[b].abs()))
        for x, r, s in zip(got, refs, slack):
            assert ((x[b].double().transpose(0, 1) - r).abs() <= 2.0 ** -8 * 1.05 * (s + r.abs()) + 1e-4).all()
