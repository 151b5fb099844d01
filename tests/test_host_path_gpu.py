"""The C++ operators (per-tile lists, C++ autograd nodes) against the Python nodes over the raw entry points (global
sort), on lists around the lengths at which the per-tile sort changes its kind (512, 2048, 8192, 16384 and beyond), with
depths spread, crowded and all equal, and with masks of every shape."""
import pytest
import torch

import util
from test_blending_edges_gpu import scene

pytestmark = pytest.mark.gpu


def run(t, cot, W, H, local, debug):
    from diff_gaussian_rasterization import GaussianRasterizationSettings, GaussianRasterizer

    dev = t["m2"].device
    eye = torch.eye(4, device=dev)
    rs = GaussianRasterizationSettings(image_height=H, image_width=W, tanfovx=0.5, tanfovy=0.5,
                                       bg=torch.tensor([0.1, 0.2, 0.3], device=dev), scale_modifier=1.0, viewmatrix=eye,
                                       projmatrix=eye, sh_degree=3, campos=torch.zeros(3, device=dev), prefiltered=False,
                                       render_geo=True, debug=debug)
    leaves = {k: t[k].clone().requires_grad_(True) for k in ("m2", "co", "rgb", "am")}
    m2abs = torch.zeros(t["m2"].shape[0], 3, device=dev, requires_grad=True)
    out = GaussianRasterizer(rs).render_gaussians(leaves["m2"], m2abs, leaves["co"], leaves["rgb"], leaves["am"],
                                                  t["depths"], t["radii"], local, None, util.cuda_args())
    torch.autograd.backward([out[0], out[5], out[6]], cot)
    return [o.detach() for o in out], [v.grad for v in leaves.values()] + [m2abs.grad]


@pytest.mark.parametrize("depths", ["spread", "crowded", "equal"])
@pytest.mark.parametrize("P", [1, 63, 511, 512, 513, 2048, 2049, 8193, 16384, 20000])
def test_lists_equal_the_global_sort(P, depths, cuda_device):
    t, cot, W, H = scene(P, 3.0, 0.02, cuda_device)
    if depths == "crowded":
        t["depths"] = 1.0 + 1e-6 * torch.floor(t["depths"] * 8)
        t["depths"][-1] = 50.0
    elif depths == "equal":
        t["depths"] = torch.full_like(t["depths"], 2.5)
    local = torch.ones(2, 2, dtype=torch.bool, device=cuda_device)
    images, grads = run(t, cot, W, H, local, False)
    want_images, want_grads = run(t, cot, W, H, local, True)
    for a, b in zip(images, want_images):
        assert torch.equal(a, b)
    for a, b in zip(grads, want_grads):
        assert util.rel_l2(a, b) <= 2e-5


@pytest.mark.parametrize("mask", ["none", "row", "corner"])
def test_masks(mask, cuda_device):
    t, cot, W, H = scene(3000, 6.0, 0.3, cuda_device)
    local = torch.zeros(2, 2, dtype=torch.bool, device=cuda_device)
    if mask == "row":
        local[1] = True
    elif mask == "corner":
        local[0, 1] = local[1, 0] = True
    images, grads = run(t, cot, W, H, local, False)
    want_images, want_grads = run(t, cot, W, H, local, True)
    for a, b in zip(images, want_images):
        assert torch.equal(a, b)
    for a, b in zip(grads, want_grads):
        assert util.rel_l2(a, b) <= 2e-5


def test_many_tiles_and_prefetch(cuda_device):
    from diff_gaussian_rasterization import GaussianRasterizer, _C

    g, cam = util.make_case(cfg=2, n=200_000, res=(1999, 1501))          # 11750 tiles: two rounds of the tile scan
    dev = cuda_device
    gd = {k: v.to(dev) for k, v in g.items()}
    local = torch.ones((cam.H + 15) // 16, (cam.W + 15) // 16, dtype=torch.bool, device=dev)
    outs = []
    for debug, ahead in ((True, False), (False, False), (False, True)):
        rast = GaussianRasterizer(util.settings_for(cam, dev, debug=debug))
        m2, _, co, radii, depths = rast.preprocess_gaussians(gd["means3D"], gd["scales"], gd["rotations"], gd["sh"],
                                                             gd["opacities"], util.cuda_args())
        if ahead:
            _C.prefetch_num_rendered(cam.H, cam.W, m2, radii, local, depths=depths)
            assert len(_C._PREFETCH) == 1
        outs.append(rast.render_gaussians(m2, None, co, gd["rgb"], gd["all_map"], depths, radii, local, None,
                                          util.cuda_args()))
    assert len(_C._PREFETCH) == 0
    for o in outs[1:]:
        for a, b in zip(o, outs[0]):
            assert torch.equal(a, b)


@pytest.mark.parametrize("n,res", [(32 * 16384, (2048, 2048)), (32 * 16384 - 1, (2048, 2048)), (32 * 16512, (2064, 2048)),
                                   (32 * 187 + 131, (265, 161)), (127, (16, 16)), (300_003, (129, 97))])
def test_counters_in_either_memory(n, res, cuda_device):
    """Gaussians and tiles around the sizes from which the tiles' counters lie in shared memory."""
    from diff_gaussian_rasterization import GaussianRasterizer

    g, cam = util.make_case(cfg=2, n=n, res=res)
    dev = cuda_device
    gd = {k: v.to(dev) for k, v in g.items()}
    local = torch.ones((cam.H + 15) // 16, (cam.W + 15) // 16, dtype=torch.bool, device=dev)
    outs = []
    for debug in (True, False):
        rast = GaussianRasterizer(util.settings_for(cam, dev, debug=debug))
        m2, _, co, radii, depths = rast.preprocess_gaussians(gd["means3D"], gd["scales"], gd["rotations"], gd["sh"],
                                                             gd["opacities"], util.cuda_args())
        outs.append(rast.render_gaussians(m2, None, co, gd["rgb"], gd["all_map"], depths, radii, local, None,
                                          util.cuda_args()))
    for a, b in zip(*outs):
        assert torch.equal(a, b)
