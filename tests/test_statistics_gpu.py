"""The statistics kernels against the tensor forms (which the CPU tests pin to the reference's method): mask lengths
around the kernels' chunks (1024 anchors, 4096 slots), rare and dense masks, ragged offset counts."""
import pytest
import torch

import util  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,n_off,seen,sel", [(1, 1, 1.0, 1.0), (255, 10, 0.9, 0.9), (256, 3, 1.0, 0.5), (2049, 10, 0.3, 0.6), (1023, 10, 0.5, 0.6), (1024, 4, 1.0, 1.0),
                                              (1025, 4, 0.02, 0.5), (5000, 7, 0.9, 0.1), (20000, 10, 0.3, 0.6),
                                              (3000, 5, 0.0, 0.5)])
def test_anchor_statistics(N, n_off, seen, sel, cuda_device):
    from cgx.densification import AnchorStatistics

    gen = torch.Generator().manual_seed(N + n_off)
    gpu, cpu = AnchorStatistics(N, n_off, cuda_device), AnchorStatistics(N, n_off, torch.device("cpu"))
    for step in range(2):
        avm = torch.rand(N, generator=gen) < seen
        slots = int(avm.sum()) * n_off
        chosen = torch.rand(slots, generator=gen) < sel
        G = int(chosen.sum())
        a = (torch.randn(G, 2 + step, generator=gen), torch.randn(slots, 1, generator=gen),
             torch.rand(G, generator=gen) < 0.7, chosen, avm)
        cpu.training_statis(*a)
        gpu.training_statis(*[x.to(cuda_device) for x in a])
    for k in ("opacity_accum", "anchor_demon", "offset_gradient_accum", "offset_denom"):
        assert torch.allclose(getattr(gpu, k).cpu(), getattr(cpu, k), rtol=2e-6, atol=1e-7), k


@pytest.mark.parametrize("P,B,track", [(1, 1, True), (255, 3, False), (257, 17, True), (100000, 4, True)])
def test_densification_statistics(P, B, track, cuda_device):
    from cgx.densification import DensificationStats

    gen = torch.Generator().manual_seed(P)
    gpu, cpu = DensificationStats(P, cuda_device, track), DensificationStats(P, torch.device("cpu"), track)
    batches = []
    for b in range(B):
        r = torch.randint(-1, 5, (P,), generator=gen, dtype=torch.int32)
        m = torch.zeros(P, 2, requires_grad=True)
        if b != 1:
            m.grad = torch.randn(P, 2, generator=gen)
        batches.append((r, m))
    cpu.update_batch(batches)
    dev = []
    for r, m in batches:
        d = torch.zeros(P, 2, device=cuda_device, requires_grad=True)
        d.grad = None if m.grad is None else m.grad.to(cuda_device)
        dev.append((r.to(cuda_device), d))
    gpu.update_batch(dev)
    assert torch.allclose(gpu.grad_accum.cpu(), cpu.grad_accum, rtol=2e-6) and torch.equal(gpu.denom.cpu(), cpu.denom)
    if track:
        assert torch.equal(gpu.max_radii2D.cpu(), cpu.max_radii2D)
