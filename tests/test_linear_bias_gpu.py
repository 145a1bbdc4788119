"""Which calls of ``nn_ops.linear`` take the column-sum bias gradient, and what they return."""
import pytest
import torch
import torch.nn.functional as F

from supergrok15_b200.ops import nn_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape,out", [((4096, 64), 8), ((1025, 4, 40), 99), ((4097, 136), 520)])
def test_gradients_match_fp64(shape, out, dtype):
    g = torch.Generator(device="cuda").manual_seed(out)
    x, w, b = (torch.randn(s, generator=g, device="cuda").to(dtype).requires_grad_() for s in (shape, (out, shape[-1]), (out,)))
    dy = torch.randn(*shape[:-1], out, generator=g, device="cuda").to(dtype)
    assert nn_ops._col_sum_bias(x, w, b)
    y = nn_ops.linear(x, w, b)
    got = torch.autograd.grad(y, (x, w, b), dy)
    ref = [t.detach().double().requires_grad_() for t in (x, w, b)]
    want = torch.autograd.grad(F.linear(*ref), ref, dy.double())
    for a, c in zip(got, want):
        # fp32 sums of 4,097 terms, one rounding to the 16-bit types (2^-9, 2^-12 relative)
        assert a.shape == c.shape and float((a.double() - c).norm() / c.norm()) < (2e-5 if dtype == torch.float32 else 4e-3)


def test_other_calls_stay_with_the_library():
    x, w, b = (torch.randn(s, device="cuda", requires_grad=True) for s in ((4096, 16), (8, 16), (8,)))
    assert nn_ops._col_sum_bias(x, w, b)
    assert not nn_ops._col_sum_bias(x[:100], w, b) and not nn_ops._col_sum_bias(x, w, None) and not nn_ops._col_sum_bias(x, w, b.detach())
    with torch.no_grad():
        assert not nn_ops._col_sum_bias(x, w, b)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert nn_ops.linear(x, w, b).dtype == torch.bfloat16
    per_sample = torch.func.vmap(lambda t: nn_ops.linear(t, w, b))(x.detach().view(2, 2048, 16))
    assert torch.allclose(per_sample.view(4096, 8), F.linear(x, w, b), atol=1e-5)
    _, jvp = torch.func.jvp(lambda t: nn_ops.linear(t, w, b), (x.detach(),), (torch.ones_like(x),))
    assert torch.allclose(jvp, torch.ones_like(x) @ w.t(), atol=1e-5)
    (gx,) = torch.autograd.grad(nn_ops.linear(x, w, b).square().sum(), x, create_graph=True)
    got = torch.autograd.grad(gx.square().sum(), (w, b))
    (gr,) = torch.autograd.grad(F.linear(x, w, b).square().sum(), x, create_graph=True)
    for a, c in zip(got, torch.autograd.grad(gr.square().sum(), (w, b))):
        assert torch.allclose(a, c, rtol=1e-4, atol=1e-3 * float(c.abs().max()))


def test_forms_that_the_library_takes():
    """A bias with a leading dimension of one, a layer without outputs, gradients of several output gradients at once, and a frozen bias's
    neighbours: same results as F.linear."""
    x, w = (torch.randn(s, device="cuda", requires_grad=True) for s in ((2, 2100, 16), (8, 16)))
    for b in (torch.randn(1, 8, device="cuda", requires_grad=True), torch.randn(8, device="cuda", requires_grad=True)):
        dy = torch.randn(3, 2, 2100, 8, device="cuda")
        y, ref = nn_ops.linear(x, w, b), F.linear(x, w, b)
        for wanted in ((x, w, b), (b,), (w,)):
            got = torch.autograd.grad(y, wanted, dy[0], retain_graph=True)
            for a, c in zip(got, torch.autograd.grad(ref, wanted, dy[0], retain_graph=True)):
                assert a.shape == c.shape
                torch.testing.assert_close(a, c, rtol=1e-5, atol=1e-5 * float(c.abs().max()))        # fp32 sums of 4,200 terms in another order
        got = torch.autograd.grad(y, (x, w, b), dy, is_grads_batched=True)
        for a, c in zip(got, torch.autograd.grad(ref, (x, w, b), dy, is_grads_batched=True)):
            torch.testing.assert_close(a, c, rtol=1e-5, atol=1e-5 * float(c.abs().max()))
    w0, b0 = torch.zeros(0, 16, device="cuda", requires_grad=True), torch.zeros(0, device="cuda", requires_grad=True)
    gx, gw, gb = torch.autograd.grad(nn_ops.linear(x, w0, b0).sum(), (x, w0, b0))
    assert gw.shape == w0.shape and gb.shape == b0.shape and not gx.any()
    assert not nn_ops._col_sum_bias(x, w0, b0) and nn_ops._col_sum_bias(x, w, torch.zeros(8, device="cuda", requires_grad=True))


# 1.5e-7 to 2.0e-7 is what PyTorch's sum of these columns is off; chains of rows were 1.9e-7, 2.1e-7 and 2.8e-7 off
@pytest.mark.parametrize("rows,out,err", [(32768, 64, 1.45e-7), (32768, 2048, 1.5e-7), (131072, 1024, 2.0e-7), (200000, 63, 2.5e-7)])
def test_column_sums_are_as_precise_as_the_librarys(rows, out, err):
    from supergrok15_b200 import _build
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(rows, out, generator=g, device="cuda")
    want = x.double().sum(0)
    got = _build.require().col_sum(x).double()
    assert float((got - want).norm() / want.norm()) < err
    acc = torch.ones(out, device="cuda")
    assert torch.equal(_build.require().col_sum(x, acc), acc) and float((acc.double() - 1 - want).norm() / want.norm()) < err + 1e-7
