"""Loss on a rendered strip: masked L1 and masked 11x11 Gaussian-window SSIM against the ground-truth strip, as the
reference computes them on every rank's local rows (utils/loss_utils.py:88-132 `pixelwise_l1_with_mask`,
`pixelwise_ssim_with_mask`; gaussian_renderer/loss_distribution.py:2835-2885 sums them and divides by the number of
pixels of the whole image times 3).  The reference runs five grouped 11x11 convolutions and a dozen element-wise
kernels forward, and autograd's transposed convolutions backward; here the forward is one kernel and the backward
is one kernel (`cgx_strip_loss_fwd` / `cgx_strip_loss_bwd`).

    l1_sum, ssim_sum = strip_loss_sums(image, gt, mask)        # device scalars, differentiable towards `image`
    Ll1, ssim_loss = l1_sum / (n_pixels * 3), ssim_sum / (n_pixels * 3)
"""
from __future__ import annotations

from diff_gaussian_rasterization import _lib


def strip_loss_sums(image, gt, mask=None):
    """(sum of mask * |image - gt|, sum of mask * SSIM map) over a (C, H, W) strip; `mask` (H, W) bool or None."""
    return tuple(_lib.host().strip_loss(image, gt, mask))


def depth_normal(depth, fx, fy, cx, cy):
    """(3, H, W) camera-space normals of a (H, W) depth image: the reference's ``render_normal`` at scale 1 without
    offsets (gaussian_renderer/__init__.py:1311-1323; utils/graphics_utils.py:87-152), differentiable towards the
    depth (this is where the plane-depth cotangent of the rasterizer comes from in training)."""
    return _lib.host().depth_normal(depth, float(fx), float(fy), float(cx), float(cy))
