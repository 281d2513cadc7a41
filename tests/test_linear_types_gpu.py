"""Linear in fp16 and fp32 (multiplied as tf32): epilogue with bias, transposed operands, column sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("rows,n_in,n_out", [(1, 8, 8), (7, 24, 40), (64, 256, 64), (130, 264, 1000), (200, 72, 12),
                                             (515, 64, 36), (1028, 768, 200), (96, 40, 33)])
def test_linear_forward_backward(dtype, rows, n_in, n_out):
    """Against 64 bits; every route of the backward is reached (n_out or rows no multiple of 16 bytes, ragged tiles)."""
    from incin_b200.core.policy import MathMode, policy_scope
    from incin_b200.ops import functional as F
    from incin_b200.ops import gemm as G
    g = torch.Generator().manual_seed(rows + n_out)
    x, w, b, dy = (torch.randn(*s, generator=g).to(dtype).cuda() for s in ((rows, n_in), (n_out, n_in), (n_out,), (rows, n_out)))
    x, w, b = (t.requires_grad_() for t in (x, w, b))
    with policy_scope(math=MathMode.FAST):
        y = F.linear(x, w, b)
        dx, dw, db = torch.autograd.grad(y, (x, w, b), dy)
    G.check_status()
    xd, wd, bd, dyd = (t.detach().double() for t in (x, w, b, dy))
    # fp16: one rounding of the result (2^-11) and fp32 sums.  tf32: factors cut to 11 bits, 2^-10 each at worst.
    u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -9
    for got, a, c, extra in ((y, xd, wd.t(), bd), (dx, dyd, wd, None), (dw, dyd.t(), xd, None)):
        ref = a @ c + (0 if extra is None else extra)
        bound = u * ref.abs() + (2.0 ** -20 if dtype == torch.float16 else u) * (a.abs() @ c.abs()) + 1e-6
        assert ((got.double() - ref).abs() <= bound).all()
    bound = 2.0 ** -11 * dyd.sum(0).abs() + 2.0 ** -20 * dyd.abs().sum(0)
    assert ((db.double() - dyd.sum(0)).abs() <= bound + 1e-6).all() and db.dtype == dtype


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(1,), (), (40,), (1, 40), (9, 1), (9, 40)])
def test_linear_bias_broadcast(dtype, shape):
    """A bias that is not one element per output column is broadcast over the result as torch does it."""
    from incin_b200.core.policy import MathMode, policy_scope
    from incin_b200.ops import functional as F
    g = torch.Generator().manual_seed(len(shape))
    x, w, b = (torch.randn(s, generator=g).to(dtype).cuda() for s in ((9, 24), (40, 24), shape))
    with policy_scope(math=MathMode.FAST):
        y = F.linear(x, w, b)
    ref = x.double() @ w.double().t() + b.double()
    # as test_linear_forward_backward: one rounding for fp16, factors cut to 11 bits for fp32
    u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -9
    bound = u * ref.abs() + (2.0 ** -20 if dtype == torch.float16 else u) * (x.double().abs() @ w.double().abs().t()) + 1e-6
    assert y.dtype == dtype and ((y.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("shape", [(39,), (41,), (0,), (1, 1, 40), (8, 40)])
def test_linear_bias_refused(dtype, shape):
    from incin_b200.core.policy import MathMode, policy_scope
    from incin_b200.ops import functional as F
    with policy_scope(math=MathMode.FAST), pytest.raises(RuntimeError):
        F.linear(torch.zeros(9, 24, dtype=dtype, device="cuda"), torch.zeros(40, 24, dtype=dtype, device="cuda"),
                 torch.zeros(shape, dtype=dtype, device="cuda"))


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("rows,n_in,n_out", [(8184, 256, 200), (4096, 64, 72), (515, 64, 36), (3001, 64, 33)])
def test_linear_gradients_repeat(dtype, rows, n_in, n_out):
    """Under ``Determinism.REQUIRED`` (asked for around the forward; the backward runs on a thread of autograd) every
    gradient repeats to the bit; bias gradients do without it."""
    from incin_b200.core.policy import Determinism, MathMode, policy_scope
    from incin_b200.ops import functional as F
    g = torch.Generator().manual_seed(rows)
    x, w, b, dy = (torch.randn(*s, generator=g).to(dtype).cuda() for s in ((rows, n_in), (n_out, n_in), (n_out,), (rows, n_out)))
    x, w, b = (t.requires_grad_() for t in (x, w, b))
    def grads(determinism):
        with policy_scope(math=MathMode.FAST, determinism=determinism):
            y = F.linear(x, w, b)
        return torch.autograd.grad(y, (x, w, b), dy)
    first = grads(Determinism.REQUIRED)
    for _ in range(12):
        assert all(torch.equal(p, q) for p, q in zip(grads(Determinism.REQUIRED), first))
        assert torch.equal(grads(Determinism.PERMITTED)[2], first[2])
    # at most 64 additions on the way of a term into its sum, each within 2^-24 of the magnitudes; one rounding to fp16
    ref = dy.double().sum(0)
    assert ((first[2].double() - ref).abs() <= 2.0 ** -11 * ref.abs() * (dtype == torch.float16) + 2.0 ** -18 * dy.double().abs().sum(0)).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("rows,n_in,n_out", [(64, 32, 40), (7, 16, 12), (9, 24, 33)])
@pytest.mark.parametrize("wanted", [(0, 1, 2), (0,), (1,), (2,)])
def test_linear_unaligned_output_gradient(dtype, rows, n_in, n_out, wanted):
    """An output gradient that starts one element into a buffer gives the same gradients as an aligned copy of it."""
    from incin_b200.core.policy import Determinism, MathMode, policy_scope
    from incin_b200.ops import functional as F
    g = torch.Generator().manual_seed(rows)
    x, w, b, dy = (torch.randn(*s, generator=g).to(dtype).cuda() for s in ((rows, n_in), (n_out, n_in), (n_out,), (rows, n_out)))
    leaves = [t.requires_grad_(i in wanted) for i, t in enumerate((x, w, b))]
    shifted = torch.zeros(dy.numel() + 1, dtype=dtype, device="cuda")
    shifted[1:] = dy.reshape(-1)
    got = []
    for d in (dy, shifted[1:].view_as(dy)):
        with policy_scope(math=MathMode.FAST, determinism=Determinism.REQUIRED):
            y = F.linear(x, w, b)
        got.append(torch.autograd.grad(y, [leaves[i] for i in wanted], d))
    assert all(torch.equal(p, q) for p, q in zip(*got))


@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32, torch.float64])
@pytest.mark.parametrize("batch,rows,cols", [(1, 1, 1), (1, 64, 64), (3, 63, 65), (2, 128, 80), (1, 1, 300), (2, 144, 48), (1, 4194400, 1), (1, 1, 4194500),
                                             (300, 5, 7), (300, 16, 8), (5, 10, 128), (1, 333, 1001), (1, 2000, 1040), (700, 40, 24)])
def test_transpose_tiles(dtype, batch, rows, cols):
    from incin_b200.ops import tensor_ops as T
    g = torch.Generator().manual_seed(rows)
    x = torch.randint(0, 255, (batch, rows, cols), generator=g).to(dtype).cuda()
    assert torch.equal(T.materialize(x.transpose(1, 2)), x.transpose(1, 2).contiguous())
    flat = torch.zeros(batch * rows * cols + 1, dtype=dtype, device="cuda")   # a base that is not 16-byte aligned
    flat[1:] = x.reshape(-1)
    odd = flat[1:].view(batch, rows, cols)
    assert torch.equal(T.materialize(odd.transpose(1, 2)), x.transpose(1, 2).contiguous())
