"""Sizes at which the v2 step's kernels change their form: scan, sort, element kernel, and the bookkeeping kernels of the bilevel step."""
import copy

import pytest
import torch

from supergrok15_b200 import optim as O
from supergrok15_b200 import _build
from supergrok15_b200.ops import sg2 as sg2_ops

from helpers import make_params, set_grads

pytestmark = pytest.mark.gpu


def _opt(params, **kw):
    torch.manual_seed(1)
    og = O.SuperGrok2(params, warmup_steps=0, warmup_ramp=1, **kw)
    with torch.no_grad():
        for blk in (og.meta_net.mamba_fwd, og.meta_net.mamba_bwd):
            blk.rope_freq.mul_(20)
        og.meta_net.expert_W1.mul_(30); og.meta_net.expert_W2.mul_(30)
    return og


def test_scan_with_a_warp_per_item_equals_the_column_form():
    """The same tensors cut into many items of 16 steps (column form) and into few long ones (a warp each): the association order of
    the chunk carries differs, the bounds are those of the many-chunk test."""
    res = []
    for chunk in (16, 4096):
        torch.manual_seed(0)
        ps = make_params([(30011,), (17, 3), (1,)], torch.float32, "cuda", 5)
        og = _opt(ps)
        og.scan_chunk_len = chunk
        for s in range(2):
            og.step(); set_grads(ps, 30 + s)
        n_items = -(-30011 // chunk) * 2
        assert (n_items > 148 * 5 * 4) == (chunk == 16)                 # items that one warp each can hold at once
        res.append([p.detach().clone() for p in ps] + [og._flat_mamba_fwd_states[0].clone(), og._flat_mamba_bwd_states[0].clone()])
    for a, b in zip(*res):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("chunk", [16, 4096])
def test_long_time_steps_with_slow_decay(chunk):
    """dt = 1e10 and exp(A_log) around 1e-11: the transition depends on their product alone, whichever of the two is large.  Column form with
    many chunks and warp form, against the CPU statement."""
    def run(device):
        ps = make_params([(30011,)], torch.float32, device, 5)
        torch.manual_seed(1)
        og = O.SuperGrok2(ps, warmup_steps=0, warmup_ramp=1)
        with torch.no_grad():
            for blk in (og.meta_net.mamba_fwd, og.meta_net.mamba_bwd):
                blk.dt_proj.weight.zero_()
                blk.dt_proj.bias.fill_(1e10)
                blk.rope_freq.zero_()
                blk.A_log.sub_(25.0)
        og.scan_chunk_len = chunk
        og.step()
        return [og._flat_mamba_fwd_states[0].double().cpu(), og._flat_mamba_bwd_states[0].double().cpu()]
    for a, b in zip(run("cuda"), run("cpu")):
        assert float(b.norm()) > 0 and float((a - b).norm() / b.norm()) < 1e-4         # fp32 recurrences of some ten steps' memory; capped time steps: 0.5 and more


@pytest.mark.parametrize("filler", [3_800_001, 9_900_001])
def test_element_kernel_parts_agree(filler):
    """A CTA of the element kernel and of the preparation takes 512 or 2,048 elements by the size of the step: tensors around those
    edges get the same values whether they are stepped alone (the form of the oracle test) or beside a large tensor."""
    sizes, res = [1, 511, 513, 2047, 2049, 8191, 8193], []
    for extra in ([], [filler]):
        ps = [make_params([(n,)], torch.float32, "cuda", 40 + i)[0] for i, n in enumerate(sizes + extra)]
        og = _opt(ps)
        og.scan_chunk_len = 512
        for s in range(2):
            og.step()
            for i, p in enumerate(ps):
                set_grads([p], 60 + i + s)
        res.append([p.detach().clone() for p in ps[: len(sizes)]] + [og._flat_gru_states[i].clone() for i in range(len(sizes))])
    for a, b in zip(*res):
        torch.testing.assert_close(a, b, rtol=1e-4, atol=2e-6)


# two segment bytes; more segments than a CTA can hold the offsets of; empty segments; one element past a tile
@pytest.mark.parametrize("sizes", [[3] * 300, [2] * 5000, [0, 5, 0, 0, 4096, 0], [4097], [4095, 1, 1]])
def test_sort_segments(sizes):
    C = _build.require()
    total = sum(sizes)
    g = torch.Generator(device="cuda").manual_seed(total)
    x = torch.randint(0, 50, (total,), generator=g, device="cuda").float() * torch.randint(0, 2, (total,), generator=g, device="cuda")
    x[:: 3] = torch.rand(x[:: 3].shape, generator=g, device="cuda")
    offs = torch.zeros(len(sizes) + 1, dtype=torch.int64)
    offs[1:] = torch.tensor(sizes).cumsum(0)
    keys0 = x.view(torch.int32).clone()
    vals0 = torch.arange(total, device="cuda", dtype=torch.int32)
    keys1, vals1 = torch.empty_like(keys0), torch.empty_like(vals0)
    hist = torch.empty(256 * C.sg2_sort_blocks(total), dtype=torch.int32, device="cuda")
    tot = torch.empty(256, dtype=torch.int32, device="cuda")
    cur = C.sg2_sort(keys0, keys1, vals0, vals1, hist, tot, offs.cuda(), len(sizes), total)
    seg = torch.repeat_interleave(torch.arange(len(sizes)), torch.tensor(sizes))
    by_key = torch.argsort(x.cpu(), stable=True)
    want = by_key[torch.argsort(seg[by_key], stable=True)]
    assert torch.equal((vals1 if cur else vals0).cpu().long(), want)


@pytest.mark.parametrize("hidden", [16, 5])
def test_pack_kernel_equals_the_statement(hidden):
    mn = O.SuperGrok2([torch.nn.Parameter(torch.zeros(4))], expert_hidden=hidden).meta_net
    with torch.no_grad():
        for p in mn.parameters():
            p.normal_(0, 0.5)
    want = sg2_ops.pack_metanet(copy.deepcopy(mn).cpu())
    got = sg2_ops.pack_metanet(mn.cuda()).cpu()
    torch.testing.assert_close(got, want, rtol=3e-7, atol=0.0)          # copies; the folded tables are fp64 sums in another order, rounded once


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_unit_vectors(dtype):
    """Unit vectors per tensor; zeros for a tensor with a non-finite entry; a tensor without length keeps its values."""
    C = _build.require()
    g = torch.Generator(device="cuda").manual_seed(2)
    ts = [torch.randn(n, generator=g, device="cuda").to(dtype) for n in (1, 8191, 8193, 40000, 33, 64, 5)]
    ts[3][39999] = float("inf"); ts[4][0] = float("nan")
    ts[5].zero_()
    ts[6].fill_(1e-15)
    offs = [0]
    for t in ts:
        offs.append(offs[-1] + t.numel())
    out = C.sg2_unit_vectors(ts, offs[:-1], offs[-1])
    for t, a, b in zip(ts, offs[:-1], offs[1:]):
        v = t.double()
        n = float(v.norm())
        want = torch.zeros_like(v) if not torch.isfinite(v).all() else v / n if n > 1e-12 else v
        torch.testing.assert_close(out[a:b].double(), want, rtol=1e-6, atol=0.0)


def test_unit_vectors_of_more_tensors_than_a_launch_takes():
    """A launch takes at most 96 tensors: the others' totals and offsets belong to the next one."""
    C = _build.require()
    g = torch.Generator(device="cuda").manual_seed(4)
    ts = [torch.randn(1 + 37 * i % 600, generator=g, device="cuda") * 10.0 ** (i % 7 - 3) for i in range(211)]
    ts[100][0] = float("nan")
    offs = torch.tensor([0] + [t.numel() for t in ts]).cumsum(0).tolist()
    out = C.sg2_unit_vectors(ts, offs[:-1], offs[-1])
    for i, (t, a, b) in enumerate(zip(ts, offs[:-1], offs[1:])):
        want = torch.zeros_like(t) if i == 100 else t / t.double().norm()
        torch.testing.assert_close(out[a:b].double(), want.double(), rtol=1e-6, atol=0.0)
