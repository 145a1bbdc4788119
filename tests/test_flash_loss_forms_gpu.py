"""Work-item counts and row lengths at which the attention backward and the cross-entropy kernels can go wrong."""
import pytest
import torch
import torch.nn.functional as F

from supergrok15_b200.ops import gemm, nn_ops

pytestmark = pytest.mark.gpu


# fewer items than CTAs, exactly one round, one item more, several rounds dealt back and forth with a partial last one; one iteration
# per item (S = 128 and the ends of the causal triangle) and many
@pytest.mark.parametrize("B,S,H,HD,causal", [(1, 128, 1, 64, False), (37, 128, 4, 128, True), (1, 128, 149, 64, True), (3, 640, 31, 64, True),
                                             (2, 1152, 17, 128, True), (2, 768, 25, 128, False), (1, 2048, 3, 128, True)])
def test_flash_backward_items(B, S, H, HD, causal):
    g = torch.Generator(device="cuda").manual_seed(S + H)
    q, k, v, do = (torch.randn(B, S, H, HD, generator=g, device="cuda").to(torch.bfloat16) for _ in range(4))
    for t in (q, k, v):
        t.requires_grad_(True)
    got = torch.autograd.grad(nn_ops.attention(q, k, v, causal, impl="tcgen05"), (q, k, v), do)
    torch.cuda.synchronize()
    gemm.check(q.device)
    again = torch.autograd.grad(nn_ops.attention(q, k, v, causal, impl="tcgen05"), (q, k, v), do)
    ref = [t.detach().float().requires_grad_(True) for t in (q, k, v)]
    want = torch.autograd.grad(nn_ops.attention_reference(*ref, causal), ref, do.float())
    for a, b, c in zip(got, want, again):
        assert torch.equal(a, c)                                        # no atomics: fixed order
        # P, dS and the results are rounded to bf16 (2^-9 each), as are O and dO in delta: under 1 % of the gradient's norm
        rel = float((a.float() - b).norm() / b.norm())
        assert rel < 1e-2, rel


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,V", [(1, 8), (4097, 16), (5, 2040), (3, 2048), (7, 2056), (2, 32008), (9000, 24)])
def test_cross_entropy_row_lengths(rows, V, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows + V)
    x = (torch.randn(rows, V, generator=g, device="cuda") * 4).to(dtype).requires_grad_(True)
    t = torch.randint(0, V, (rows,), generator=g, device="cuda")
    t[1::5] = -100
    xr = x.detach().double().requires_grad_(True)
    loss, want = nn_ops.cross_entropy(x, t), F.cross_entropy(xr, t, ignore_index=-100)
    # fp32 exponentials and sums of up to 32,008 terms: 2^-23 times a few tens of roundings
    assert abs(float(loss) - float(want)) < 1e-5 * max(1.0, float(want))
    gx, = torch.autograd.grad(loss * rows, x)                           # times rows: 16-bit gradients stay in the normal range
    gr, = torch.autograd.grad(want * rows, xr)
    rel = float((gx.double() - gr).norm() / gr.norm())
    assert rel < {torch.float32: 1e-5, torch.bfloat16: 4e-3, torch.float16: 2e-3}[dtype], rel
