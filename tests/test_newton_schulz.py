"""The grouped Newton-Schulz iteration of Muon: tile order of its symmetric products (CPU) and results for lists of matrices (GPU)."""
import pytest
import torch

from supergrok15_b200 import _build
from supergrok15_b200.ops import gemm, muon, oracle


@pytest.mark.parametrize("bn", [64, 128, 256])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 255, 256, 257, 300, 512, 777, 2048])
def test_symmetric_tiles_cover_every_element_once(n, bn):
    C = _build.load()
    if C is None:
        pytest.skip("extension not built")
    hit = torch.zeros(n, n, dtype=torch.int32)
    for m0, n0, mirror in C.ns_sym_tiles(n, bn):
        if m0 >= n or n0 >= n:
            continue
        hit[m0:m0 + 128, n0:n0 + bn] += 1
        if mirror:
            assert m0 + 128 <= n0                       # strictly above the diagonal: its transpose is a tile that nobody computes
            hit[n0:n0 + bn, m0:m0 + 128] += 1
    assert bool((hit == 1).all())


# a lone tiny matrix, edges of the 64 / 128 / 256 tiles and of the 8-element row padding, tall, wide and square matrices mixed, enough
# matrices of a shape for every tile width
LISTS = [[(1, 1)], [(3, 40), (40, 3), (8, 8)], [(64, 64), (65, 64), (64, 65), (129, 127)], [(256, 256)] * 3 + [(768, 256), (256, 1024), (255, 257)],
         [(512, 512)] * 12 + [(1536, 512), (512, 2048)], [(1024, 520)] * 5 + [(520, 1032)] * 3, [(1032, 2048)] * 2,
         [(72 + 8 * i, 136) for i in range(9)]]          # more shapes than the small parameter block holds


@pytest.mark.gpu
@pytest.mark.parametrize("shapes", LISTS, ids=lambda s: f"{len(s)}x{s[0][0]}x{s[0][1]}")
def test_grouped_iteration_matches_the_fp64_iteration(shapes):
    torch.manual_seed(len(shapes) + shapes[0][0])
    C = _build.require()
    mats = [torch.randn(s, device="cuda") for s in shapes]
    inv = torch.stack([1.0 / (m.norm() + 1e-7) for m in mats])
    outs = C.newton_schulz(mats, inv, 5, *muon.NS_COEFFS, gemm._err_flag(mats[0].device))
    gemm.check()
    for m, i, o in zip(mats, inv, outs):
        ref = oracle.newton_schulz((m * i).double(), 5)
        assert o.shape == ref.shape
        # three bf16-rounded operands per iteration; the bound is the one of the single-matrix test
        assert float((o - ref).norm() / ref.norm()) < 0.06
        lone = gemm.newton_schulz(m * i, 5, muon.NS_COEFFS)
        assert float((o - lone).norm() / ref.norm()) < 1e-2          # the tile width may differ, the products do not


@pytest.mark.gpu
def test_long_lists_go_in_runs(monkeypatch):
    torch.manual_seed(0)
    ps, gs = [torch.randn(136, 72, device="cuda") for _ in range(5)], [torch.randn(136, 72, device="cuda") for _ in range(5)]
    outs = []
    for run in (1 << 28, 2 * 136 * 72, 1):
        monkeypatch.setattr(muon, "NS_RUN_ELEMS", run)
        p, b = [t.clone() for t in ps], [torch.zeros_like(t) for t in ps]
        muon.muon_step(p, gs, b, 0.02, 0.95, 0.1, 5)
        outs.append(p)
    for o in outs[1:]:
        assert all(torch.equal(x, y) for x, y in zip(outs[0], o))


@pytest.mark.parametrize("shape", [(4096, 1), (1, 4096), (1000, 9), (64, 64), (300, 5), (8, 2048)])
def test_runs_bound_the_workspace_that_padding_makes(shape, monkeypatch):
    """What a run allocates, row padding and the dense copies of padded results included, stays within 12 bytes per element of the bound."""
    r, c = shape
    k, up = min(r, c), lambda n, m: -(-n // m) * m
    each = 2 * 2 * r * up(c, 8) + 2 * 2 * k * up(k, 8) + 4 * r * up(c, 4) + (4 * r * c if c % 4 else 0)
    monkeypatch.setattr(muon, "NS_RUN_ELEMS", 1 << 16)
    runs = list(muon._runs([shape] * 50))
    assert [i for i, _ in runs] == [0] + [j for _, j in runs[:-1]] and runs[-1][1] == 50
    assert all((j - i) * each <= 12 << 16 or j == i + 1 for i, j in runs)
    assert all((j - i + 1) * each > (12 << 16) - 12 * (j - i + 1) for i, j in runs[:-1])             # and no run is shorter than it has to be
