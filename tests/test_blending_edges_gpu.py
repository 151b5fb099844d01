"""Blending on lists whose length sits at the edges of what the kernels take at a time (a queue of 32, a stretch of
256), with small and with block-filling splats, transparent and saturating: the queued walks against the plain ones,
and the backward through the table of rows against the backward straight into the tensors."""
import pytest
import torch

import util  # noqa: F401

pytestmark = pytest.mark.gpu


def scene(P, spread, opacity, dev):
    gen = torch.Generator().manual_seed(P)
    W = H = 32                                                   # 2 x 2 tiles; everything lies around the middle
    m2 = 16 + spread * torch.randn(P, 2, generator=gen)
    inv = 1.0 / (0.3 + 4.0 * torch.rand(P, 2, generator=gen) * spread)
    off = (torch.rand(P, generator=gen) - 0.5) * (inv[:, 0] * inv[:, 1]).sqrt()
    co = torch.stack([inv[:, 0], off, inv[:, 1], opacity * (0.2 + 0.8 * torch.rand(P, generator=gen))], 1)
    t = dict(m2=m2, depths=1 + torch.rand(P, generator=gen), radii=torch.full((P,), 40, dtype=torch.int32),
             co=co, rgb=torch.rand(P, 3, generator=gen), am=torch.randn(P, 5, generator=gen))
    cot = [torch.randn(n, H, W, generator=gen).to(dev) for n in (3, 5, 1)]
    return {k: v.to(dev).contiguous() for k, v in t.items()}, cot, W, H


def run(t, cot, W, H, geo, variant, table):
    from diff_gaussian_rasterization import _C, _lib

    l = _lib.lib()
    dev = t["m2"].device
    local = torch.ones(2, 2, dtype=torch.bool, device=dev)
    bg = torch.tensor([0.1, 0.2, 0.3], device=dev)
    l.cgx_set_render_variant(variant)
    try:
        out = _C.render_gaussians(bg, H, W, t["m2"], t["depths"], t["radii"], t["co"], t["rgb"], local, None, None, 0.5,
                                  0.5, t["am"], geo, True, {})
        P, R = t["m2"].shape[0], out[0]
        g = _C.geometry_layout(P).views(out[8])
        b, im = _C.binning_layout(R).views(out[9]), _C.image_layout(W * H, 4).views(out[10])
        grads = [torch.full((P, n), float("nan"), device=dev) for n in (2, 3, 4, 3, 5)]
        ws = torch.empty(l.cgx_render_bwd_workspace_bytes(P), dtype=torch.uint8, device=dev)
        p = lambda x: x.data_ptr()  # noqa: E731
        st = l.cgx_render_bwd_table(P, W, H, 0.5, 0.5, p(im["ranges"]), p(b["point_list"]), p(bg), p(g["records"]),
                                    p(out[6]), p(im["accum_alpha"]), p(im["n_contrib"]), p(local), *map(p, cot),
                                    int(geo), *map(p, grads), 2, p(g["tiles_touched"]) if table else None,
                                    p(ws) if table else None, ws.numel() if table else 0, _lib.current_stream_ptr())
        assert st == 0
        torch.cuda.synchronize()
    finally:
        l.cgx_set_render_variant(1)
    return [out[k] for k in (1, 2, 3, 4, 5, 6, 7)], grads


@pytest.mark.parametrize("geo", [True, False])
@pytest.mark.parametrize("spread,opacity", [(4.0, 0.02), (1.0, 0.9), (12.0, 0.3)])
@pytest.mark.parametrize("P", [1, 31, 32, 33, 64, 255, 256, 257, 513])
def test_queued_walks_equal_plain_walks(P, spread, opacity, geo, cuda_device):
    t, cot, W, H = scene(P, spread, opacity, cuda_device)
    images, grads = run(t, cot, W, H, geo, 1, True)
    plain_images, plain_grads = run(t, cot, W, H, geo, 0, False)
    _, direct_grads = run(t, cot, W, H, geo, 1, False)
    for a, b in zip(images, plain_images):
        assert torch.equal(a, b)
    for a, b, c in zip(grads, plain_grads, direct_grads):
        assert torch.isfinite(a).all()
        if not geo and a.shape[1] == 5:
            assert not a.any() and not c.any()
            continue
        assert util.rel_l2(a, b) <= 2e-5 and util.rel_l2(c, b) <= 2e-5
