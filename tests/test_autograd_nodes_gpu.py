"""The C++ autograd nodes of ``nn_ops`` against the Python functions they stand in for: same results bit for bit, and the same behaviour
where an autograd function is looked into (saved-tensor hooks, in-place changes, second backward, frozen inputs, transforms)."""
import contextlib

import pytest
import torch

from supergrok15_b200.ops import nn_ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _t(*shape, dtype=torch.bfloat16, grad=True):
    g = torch.Generator(device=DEV).manual_seed(sum(shape))
    return torch.randn(*shape, generator=g, device=DEV).to(dtype).requires_grad_(grad)


def _ops():
    ang = torch.rand(8, 32, device=DEV)
    tgt = torch.randint(0, 64, (40,), device=DEV)
    tgt[3] = -100
    return {
        "layer_norm": (lambda x, r, w, b: nn_ops.layer_norm(x, r, w, b), [_t(33, 256), _t(33, 256), _t(256), _t(256)]),
        "layer_norm_plain": (lambda x, w: nn_ops.layer_norm(x, None, w, None), [_t(17, 4, 128, dtype=torch.float32), _t(128, dtype=torch.float32)]),
        "layer_norm_strided": (lambda x, w, b: nn_ops.layer_norm(x.transpose(0, 1), None, w, b), [_t(9, 5, 64), _t(64), _t(64)]),
        "rms_norm": (lambda x, r, w: nn_ops.rms_norm(x, r, w), [_t(7, 264), _t(7, 264), _t(264)]),
        "norm_residual": (lambda x, r, w: nn_ops.norm_residual(x, r, w, None, rms=True), [_t(31, 512), _t(31, 512), _t(512)]),
        "attention_small": (lambda q: nn_ops.attention_small(q, 2), [_t(11, 4, 3 * 128)]),
        "cross_entropy": (lambda x: nn_ops.cross_entropy(x, tgt), [_t(40, 64)]),
        "gelu": (lambda x: nn_ops.gelu(x), [_t(16, 64)]),
        "swiglu": (lambda a, b: nn_ops.swiglu(a, b), [_t(16, 64), _t(8, 128).detach().view(16, 64).requires_grad_()]),
        "rope": (lambda x: nn_ops.rope(x, ang.cos(), ang.sin()), [_t(2, 8, 3, 64)]),
        "flash": (lambda q, k, v: nn_ops.attention(q, k, v, True, impl="tcgen05"), [_t(1, 128, 2, 64), _t(1, 128, 2, 64), _t(2, 64, 2, 64).detach().view(1, 128, 2, 64).requires_grad_()]),
    }


@contextlib.contextmanager
def _python_nodes(monkeypatch):
    with monkeypatch.context() as m:
        m.setattr(nn_ops, "_cpp_node", lambda *a: False)
        yield


def _run(fn, args, needed=None):
    out = fn(*args)
    outs = out if isinstance(out, tuple) else (out,)
    grads = [torch.ones_like(o) * (0.5 + k) for k, o in enumerate(outs)]
    wanted = [a for a in args if a.requires_grad]
    return outs, torch.autograd.grad(outs, wanted, grads, allow_unused=True)


@pytest.mark.parametrize("name", list(_ops()) if torch.cuda.is_available() else ["none"])
def test_same_as_the_python_function(name, monkeypatch):
    fn, args = _ops()[name]
    assert nn_ops._cpp_node(*args)
    outs, grads = _run(fn, args)
    with _python_nodes(monkeypatch):
        outs_p, grads_p = _run(fn, args)
    for a, b in zip((*outs, *grads), (*outs_p, *grads_p)):
        assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)
    # frozen inputs: the others' gradients stay what they were, nothing is returned for the frozen one
    if len(args) > 1:
        frozen = [args[0], *[a.detach() for a in args[1:]]]
        assert torch.equal(_run(fn, frozen)[1][0], grads[0])
    with torch.no_grad():
        free = fn(*args)
        assert not (free[0] if isinstance(free, tuple) else free).requires_grad


@pytest.mark.parametrize("name", list(_ops()) if torch.cuda.is_available() else ["none"])
def test_saved_tensors_can_be_packed(name):
    fn, args = _ops()[name]
    _, want = _run(fn, args)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(), lambda t: t.cuda()):
        out = fn(*args)
    outs = out if isinstance(out, tuple) else (out,)
    got = torch.autograd.grad(outs, args, [torch.ones_like(o) * (0.5 + k) for k, o in enumerate(outs)])
    assert packed and all(torch.equal(a, b) for a, b in zip(got, want))


def test_in_place_changes_second_backward_and_transforms():
    x, w = _t(8, 64), _t(64)
    y = nn_ops.gelu(x * 1.0)
    y.sum().backward(retain_graph=True)
    y.sum().backward()
    with pytest.raises(RuntimeError, match="second time|already been freed"):
        y.sum().backward()
    a = x * 1.0
    y = nn_ops.gelu(a)
    a.add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace"):
        y.sum().backward()
    assert nn_ops._cpp_node(x, w)
    seen = []
    torch.func.vmap(lambda t: (seen.append(nn_ops._cpp_node(t)), t)[1])(torch.zeros(2, 3, device=DEV))
    torch.func.jvp(lambda t: (seen.append(nn_ops._cpp_node(t)), t)[1], (torch.zeros(2, device=DEV),), (torch.ones(2, device=DEV),))
    with nn_ops.grad_sink(True):
        seen.append(nn_ops._cpp_node(x))
    assert seen == [False, False, False]


def test_flash_backward_gets_the_time_out_flag_itself():
    """The flag is no saved tensor: packing hooks do not see it, and a check that clears it between forward and backward is no in-place change."""
    from supergrok15_b200.ops import gemm
    fn, args = _ops()["flash"]
    _, want = _run(fn, args)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.dtype) or t, lambda t: t):
        out = fn(*args)
    flag = gemm._err_flag(args[0].device)
    version = flag._version
    flag.zero_()
    got = torch.autograd.grad(out, args, torch.full_like(out, 0.5))
    assert torch.int32 not in packed and flag._version == version + 1
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    out = fn(*args)
    flag.zero_()                                           # without hooks
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(out, args, torch.full_like(out, 0.5)), want))
