"""Strip loss and depth normals at sizes around what a warp or a block takes (32 columns, segments of rows, 32 x 32
pixels), against the tensor forms in float64."""
import pytest
import torch

import util  # noqa: F401
from util_loss import reference_normal, reference_sums

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 1, 1), (1, 5, 31), (3, 10, 32), (1, 11, 33), (2, 128, 64), (3, 129, 65), (1, 700, 5)])
def test_strip_loss(shape, cuda_device):
    from cgx.strip_loss import strip_loss_sums

    gen = torch.Generator().manual_seed(sum(shape))
    gt = torch.rand(shape, generator=gen).to(cuda_device)
    x = (gt.cpu() * 0.6 + 0.4 * torch.rand(shape, generator=gen)).to(cuda_device).requires_grad_(True)
    mask = (torch.rand(shape[1:], generator=gen) > 0.2).to(cuda_device)
    mask[0, 0] = True
    l1, ss = strip_loss_sums(x, gt, mask)
    (0.8 * l1 - 0.2 * ss).backward()
    x64 = x.detach().double().requires_grad_(True)
    rl1, rss = reference_sums(x64, gt.double(), mask)
    (0.8 * rl1 - 0.2 * rss).backward()
    n = x.numel()
    assert abs(l1.item() - rl1.item()) <= 1e-5 * n ** 0.5 and abs(ss.item() - rss.item()) <= 2e-5 * n ** 0.5
    assert ((x.grad.double() - x64.grad).norm() / x64.grad.norm()).item() <= 1e-4


@pytest.mark.parametrize("H,W", [(31, 32), (32, 33), (33, 31), (64, 65), (3, 97), (97, 3)])
def test_depth_normal(H, W, cuda_device):
    from cgx.strip_loss import depth_normal

    gen = torch.Generator().manual_seed(H * 1000 + W)
    d = (20.0 + torch.rand(H, W, generator=gen)).to(cuda_device).requires_grad_(True)
    cot = torch.randn(3, H, W, generator=gen).to(cuda_device)
    n = depth_normal(d, 0.8 * W, 0.9 * W, W / 2, H / 2)
    (n * cot).sum().backward()
    d64 = d.detach().double().requires_grad_(True)
    n64 = reference_normal(d64, 0.8 * W, 0.9 * W, W / 2, H / 2)
    (n64 * cot.double()).sum().backward()
    assert (n.double() - n64).abs().max().item() <= 2e-5
    assert ((d.grad.double() - d64.grad).norm() / d64.grad.norm()).item() <= 1e-3
