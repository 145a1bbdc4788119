"""What ``SuperGrok2.bilevel_step`` leaves in the parameters' gradients when a backward writes into storage that it reuses."""
import os
import socket

import pytest
import torch
import torch.nn as nn

from supergrok15_b200 import optim as O


def _rank(_, port, out):
    import torch.distributed as dist
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
    dist.init_process_group("gloo", rank=0, world_size=1)
    res = {}
    for views in (False, True):
        torch.manual_seed(0)
        model = nn.Sequential(nn.Linear(6, 5), nn.Tanh(), nn.Linear(5, 3))
        net = nn.parallel.DistributedDataParallel(model, gradient_as_bucket_view=views)
        opt = O.SuperGrok2(model.parameters())
        meta = torch.optim.SGD(opt.meta_net.parameters(), lr=0.0)
        crit = nn.CrossEntropyLoss()
        x, y = [torch.randn(16, 6) for _ in range(4)], [torch.randint(0, 3, (16,)) for _ in range(4)]
        for k in (0, 1):                                   # from the second backward on the gradients live in the reducer's buckets
            net.zero_grad()
            crit(net(x[k]), y[k]).backward()
        before = [p.grad.clone() for p in model.parameters()]
        opt.bilevel_step(net, x[1], y[1], x[2], y[2], crit, meta)
        res[views] = dict(kept=[torch.equal(a, p.grad) for a, p in zip(before, model.parameters())],
                          meta=[p.grad.clone() for p in opt.meta_net.parameters() if p.grad is not None])
    torch.save(res, out)
    dist.destroy_process_group()


@pytest.mark.dist
def test_bilevel_step_keeps_gradients_that_live_in_reused_buffers(tmp_path):
    """DistributedDataParallel with ``gradient_as_bucket_view`` fills the same buckets in every backward: the training gradients and the
    meta-gradient are those of the run whose gradients have storage of their own."""
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        port = s.getsockname()[1]
    torch.multiprocessing.spawn(_rank, args=(port, str(tmp_path / "r.pt")), nprocs=1)
    res = torch.load(tmp_path / "r.pt")
    for views in (False, True):
        assert all(res[views]["kept"]), views
    assert len(res[True]["meta"]) > 0
    for a, b in zip(res[False]["meta"], res[True]["meta"]):
        assert torch.equal(a, b)


def test_copies_are_exact_and_own_their_storage():
    from supergrok15_b200.optim.supergrok2 import _copies
    odd = torch.tensor([0.0, -0.0, float("inf"), float("-inf"), float("nan"), 1e-45, 3e38])
    ts = [odd, odd.double(), odd.bfloat16(), odd.half(), torch.randn(3, 4).t(), torch.zeros(0), torch.eye(3).to_sparse(), torch.nn.Parameter(torch.ones(2))]
    for a, b in zip(ts, _copies(ts)):
        assert a.dtype == b.dtype and a.shape == b.shape and a.layout == b.layout and not b.requires_grad
        if a.layout == torch.strided:
            assert a.stride() == b.stride() and (a.numel() == 0 or a.data_ptr() != b.data_ptr())
            number = ~a.isnan()                            # which NaN it is does not matter
            assert torch.equal(number, ~b.isnan()) and torch.equal(a[number], b[number]) and torch.equal(torch.signbit(a[number]), torch.signbit(b[number]))
        else:
            assert torch.equal(a.to_dense(), b.to_dense())
