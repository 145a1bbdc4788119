"""Row widths, row counts and alignments at which the norm and short-attention kernels change their form."""
import pytest
import torch
import torch.nn.functional as F

from supergrok15_b200.ops import nn_ops

pytestmark = pytest.mark.gpu


def _close(a, b, dtype, sums=False):
    # fp32: sums of up to 3072 products; 16 bits: one rounding of the result and one of the stored sum x + r (2^-9 each, times a few
    # units); parameter gradients add up to 40,000 rows before their one rounding
    rel = float((a.double() - b).norm() / b.norm())
    assert rel < (3e-6 if dtype == torch.float32 else 1e-2 if sums else 5e-3), rel


# one vector, a partial warp, whole warps, a partial last warp of a row, the most warps per row; too few rows for the four-row form,
# enough, and a remainder; widths of half a vector (the general kernel)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,D", [(1, 8), (3, 64), (5, 264), (17, 768), (2369, 2048), (40001, 72), (9475, 256), (4739, 520), (131, 3072), (2400, 1544), (33, 132), (1190, 3000)])
@pytest.mark.parametrize("rms,res", [(False, True), (False, False), (True, True)])
def test_norm_matches_fp64(rows, D, rms, res, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows + D)
    x, r, dy, dzo = (torch.randn(rows, D, generator=g, device="cuda").to(dtype) for _ in range(4))
    w, b = ((1 + torch.randn(D, generator=g, device="cuda") * 0.1).to(dtype) for _ in range(2))
    leaves = [t.requires_grad_() for t in ([x, r, w] if rms else [x, r, w, b] if res else [x, w, b])]
    ref = [t.detach().double().requires_grad_() for t in leaves]
    if rms:
        y, z = nn_ops.norm_residual(x, r, w, None, 1e-5, rms=True)
        got = torch.autograd.grad((y, z), leaves, (dy, dzo))
        zr = ref[0] + ref[1]
        if dtype != torch.float32:
            zr = zr + (z.detach().double() - zr.detach())               # the stored (rounded) sum is what the norm sees
        yr = zr * torch.rsqrt(zr.square().mean(-1, keepdim=True) + 1e-5) * ref[2]
        want = torch.autograd.grad((yr, zr), ref, (dy.double(), dzo.double()))
    else:
        y = nn_ops.layer_norm(x, r if res else None, w, b)
        got = torch.autograd.grad(y, leaves, dy)
        zr = ref[0] + ref[1] if res else ref[0]
        if dtype != torch.float32 and res:
            zr = zr + ((x.detach() + r.detach()).double() - zr.detach())
        yr = F.layer_norm(zr, (D,), ref[-2], ref[-1], 1e-5)
        want = torch.autograd.grad(yr, ref, dy.double())
    _close(y.detach(), yr.detach(), dtype)
    for k, (a, c) in enumerate(zip(got, want)):
        _close(a, c, dtype, sums=a.dim() == 1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,H,hd,off", [(1, 4, 1, 64, 0), (37, 4, 3, 64, 0), (129, 4, 5, 32, 0), (11, 8, 3, 64, 0), (33, 8, 1, 32, 0), (7, 4, 3, 64, 2), (5, 8, 3, 32, 2)])
def test_short_attention_matches_fp64(B, S, H, hd, off, causal, dtype):
    """``off``: the input starts that many elements into a buffer, which breaks the 16-byte alignment that the wide loads need."""
    g = torch.Generator(device="cuda").manual_seed(B + S)
    n = B * S * 3 * H * hd
    qkv = torch.randn(n + off, generator=g, device="cuda").to(dtype)[off:].view(B, S, 3 * H * hd).requires_grad_()
    do = torch.randn(B, S, H * hd, generator=g, device="cuda").to(dtype)
    o = nn_ops.attention_small(qkv, H, causal)
    (got,) = torch.autograd.grad(o, qkv, do)
    ref = qkv.detach().double().requires_grad_()
    orf = nn_ops.attention_small_reference(ref, H, causal)
    (want,) = torch.autograd.grad(orf, ref, do.double())
    _close(o.detach(), orf.detach(), dtype)
    _close(got, want, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("S,hd", [(4, 64), (4, 32), (8, 64), (8, 32)])
@pytest.mark.parametrize("off", [1, 3, 4, 7])
def test_short_attention_from_any_element_of_a_buffer(S, hd, off, dtype):
    """Input and output gradient start ``off`` elements into a buffer: every alignment that a contiguous view can have."""
    B, H = 9, 3
    g = torch.Generator(device="cuda").manual_seed(off + S)
    n = B * S * H * hd
    qkv, do = (torch.randn(m + off, generator=g, device="cuda").to(dtype)[off:].view(B, S, -1) for m in (3 * n, n))
    o = nn_ops.attention_small(qkv.requires_grad_(), H, True)
    (got,) = torch.autograd.grad(o, qkv, do)
    ref = qkv.detach().double().requires_grad_()
    orf = nn_ops.attention_small_reference(ref, H, True)
    (want,) = torch.autograd.grad(orf, ref, do.double())
    _close(o.detach(), orf.detach(), dtype)
    _close(got, want, dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 512, 132])
@pytest.mark.parametrize("off", [1, 2, 3, 4])
@pytest.mark.parametrize("which", ["x", "r", "w", "b", "dy", "all"])
def test_norm_from_any_element_of_a_buffer(which, off, D, dtype):
    """Each operand, and all of them, start ``off`` elements into a buffer: every alignment that a contiguous view can have."""
    rows = 37
    gen = torch.Generator(device="cuda").manual_seed(off + D)

    def make(name, *shape):
        o = off if which in (name, "all") else 0
        n = 1
        for k in shape:
            n *= k
        return torch.randn(n + o, generator=gen, device="cuda").to(dtype)[o:].view(shape)
    x, r, dy = (make(k, rows, D) for k in ("x", "r", "dy"))
    w, b = make("w", D), make("b", D)
    leaves = [t.requires_grad_() for t in (x, r, w, b)]
    y = nn_ops.layer_norm(x, r, w, b)
    got = torch.autograd.grad(y, leaves, dy)
    ref = [t.detach().double().requires_grad_() for t in leaves]
    zr = ref[0] + ref[1]
    zr = zr + ((x.detach() + r.detach()).double() - zr.detach())          # the stored sum is what the norm sees
    yr = F.layer_norm(zr, (D,), ref[2], ref[3], 1e-5)
    _close(y.detach(), yr.detach(), dtype)
    for a, c in zip(got, torch.autograd.grad(yr, ref, dy.double())):
        _close(a, c, dtype, sums=a.dim() == 1)
    y, z = nn_ops.norm_residual(x, r, w, None, 1e-5, rms=True)
    got = torch.autograd.grad((y, z), leaves[:3], (dy, dy))
    yr = zr * torch.rsqrt(zr.square().mean(-1, keepdim=True) + 1e-5) * ref[2]
    for a, c in zip(got, torch.autograd.grad((yr, zr), ref[:3], (dy.double(), dy.double()))):
        _close(a, c, dtype, sums=a.dim() == 1)


@pytest.mark.parametrize("rows,D,y_err,w_err", [(300, 3072, 6.9e-8, 1.2e-7), (10000, 3072, 6.9e-8, 1.45e-7), (32000, 1028, 6.9e-8, 1.55e-7)])
def test_norm_sums_do_not_grow_one_by_one(rows, D, y_err, w_err):
    """fp32 sums over the warps of a row, the rows of a CTA and the CTAs' partial rows are added in groups.  An output is a product of
    three factors (6.3e-8 with an exact sum of squares; 7.4e-8 when 24 warps' sums are added one after the other), a weight gradient the sum of
    ``rows`` products (1.06e-7, 1.28e-7 and 1.37e-7 here; 1.43e-7 for 300 rows with chains, and growing)."""
    g = torch.Generator(device="cuda").manual_seed(rows)
    x, r, dy = (torch.randn(rows, D, generator=g, device="cuda") for _ in range(3))
    w = 1 + 0.1 * torch.randn(D, generator=g, device="cuda")
    leaves = [t.requires_grad_() for t in (x, r, w)]
    y, z = nn_ops.norm_residual(x, r, w, None, 1e-5, rms=True)
    got = torch.autograd.grad((y, z), leaves, (dy, dy))[2].double()
    zr = z.detach().double()
    xh = zr * torch.rsqrt(zr.square().mean(-1, keepdim=True) + 1e-5)
    yr, want = xh * w.detach().double(), (xh * dy.double()).sum(0)
    assert float((y.detach().double() - yr).norm() / yr.norm()) < y_err
    assert float((got - want).norm() / want.norm()) < w_err
