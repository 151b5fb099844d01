"""The work that is timed: what a trainer or a renderer built on this package asks of it, pass by pass, through the
public entry points (`diff_gaussian_rasterization`, `cgx.batched`, `cgx.plane_map`, `cgx.strip_loss`,
`cgx.densification`, `cgx.runtime`).

Kinds of pass:
  train   one optimisation step of the rasterizer: preprocess of the Gaussians for the batch's cameras with their plane
          descriptors, rendering of every camera, one backward pass over the batch; upstream gradients N(0,1)
  step    the same through `cgx.runtime.TrainingStep`, with the densification statistics
  band    the share of one rank of a distributed job between its two exchanges: a band of tile rows of one camera,
          rendered from the records that were received for it, and its backward pass
  eval    images for evaluation or a fly-through: forward only, no graph
  filter  the visibility test of the anchors for the batch's cameras that precedes every training iteration
  loss    the loss on a rendered strip (masked L1 and SSIM, normals from depth) and its gradient
  stats   the anchor statistics that the densifier reads, updated after every iteration

Sizes follow `cgx.synthetic.config` (its five configurations) and the ragged sizes of real captures; scenes are made
on the GPU by the same generator (`cgx.synthetic.make_gaussians`) from the seed.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("citygs-x_b200"))

from cgx import synthetic as S  # noqa: E402
from cgx.batched import preprocess_gaussians_batched  # noqa: E402
from cgx.densification import AnchorStatistics  # noqa: E402
from cgx.plane_map import plane_map  # noqa: E402
from cgx.runtime import TrainingStep, make_cuda_args  # noqa: E402
from cgx.strip_loss import depth_normal, strip_loss_sums  # noqa: E402
from diff_gaussian_rasterization import GaussianRasterizationSettings, GaussianRasterizer  # noqa: E402


def listed():
    return [
        # the smallest step anyone runs (tests, tutorials, the first minutes on a small capture): launches and host work
        dict(name="train_tiny", kind="train", gaussians=50_000, cameras=1, width=256, height=144, scene="box",
             half=50.0, top=20.0, splat=1.0, geo=True),
        # odd sizes: a capture whose images are no multiple of the tile, two cameras a step
        dict(name="train_ragged", kind="train", gaussians=333_337, cameras=2, width=1237, height=823, scene="box",
             half=70.0, top=25.0, splat=1.0, geo=True),
        # the single-GPU configuration: one Full-HD camera a step
        dict(name="train_hd", kind="train", gaussians=1_000_000, cameras=1, width=1920, height=1080, scene="box",
             half=100.0, top=30.0, splat=1.0, geo=True),
        # the first thousands of iterations: few and large splats, the geometry terms still switched off
        dict(name="train_early", kind="train", gaussians=150_000, cameras=2, width=1280, height=720, scene="box",
             half=60.0, top=20.0, splat=4.0, geo=False),
        # the data-parallel configuration on one GPU: 6 M Gaussians, a batch of eight cameras
        dict(name="train_batch", kind="train", gaussians=6_000_000, cameras=8, width=1600, height=1200, scene="box",
             half=300.0, top=40.0, splat=1.0, geo=True),
        # the large aerial city: clustered Gaussians, 4K views from above
        dict(name="train_city_4k", kind="train", gaussians=20_000_000, cameras=2, width=3840, height=2160,
             scene="city", half=600.0, top=1.0, splat=1.0, geo=True),
        # the step driver with the densification statistics
        dict(name="step_densify", kind="step", gaussians=400_000, cameras=4, width=800, height=600, scene="box",
             half=80.0, top=25.0, splat=1.0, geo=True),
        # a rank of a distributed job: the middle half of a camera's tile rows
        dict(name="band_half", kind="band", gaussians=3_000_000, cameras=1, width=1600, height=1200, scene="box",
             half=300.0, top=40.0, splat=1.0, geo=True, rows=0.5),
        # evaluation images
        dict(name="eval_4k", kind="eval", gaussians=4_000_000, cameras=1, width=3840, height=2160, scene="box",
             half=250.0, top=40.0, splat=1.0, geo=True),
        # anchors of a city against the eight cameras of a batch
        dict(name="filter_batch", kind="filter", gaussians=2_000_000, cameras=8, width=1600, height=1200, scene="box",
             half=300.0, top=40.0, splat=1.0, geo=True),
        # loss on a camera's full image, with a mask
        dict(name="loss_image", kind="loss", width=1600, height=1200, mask=True),
        # statistics of a model of 500 k anchors with ten Gaussians each
        dict(name="stats_anchors", kind="stats", anchors=500_000, offsets=10, seen=0.3, selected=0.6),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "train", "step", "band", "eval", "eval", "filter", "loss", "stats"])
    if kind == "stats":
        return dict(kind=kind, anchors=int(_log(rng, 10_000, 2_000_000)), offsets=rng.choice([5, 10]),
                    seen=round(rng.uniform(0.05, 0.9), 3), selected=round(rng.uniform(0.3, 0.9), 3))
    pixels, aspect = _log(rng, 256 * 144, 3840 * 2160), rng.uniform(1.2, 2.0)
    width = max(32, int(math.sqrt(pixels * aspect)))
    height = max(32, int(pixels / width))
    if kind == "loss":
        return dict(kind=kind, width=width, height=height, mask=rng.random() < 0.5)
    n = int(_log(rng, 20_000, 600_000 if kind == "step" else 6_000_000))
    most = min(8, 16_000_000 // (width * height), 32_000_000 // n)
    cameras = 1 if kind in ("band", "eval") else max(1, min(4 if kind == "step" else 8, rng.randint(1, max(1, most))))
    half = 0.5 * math.sqrt(n / _log(rng, 5.0, 25.0))          # 5 to 25 Gaussians per square metre
    city = kind in ("train", "eval") and n >= 1_000_000 and rng.random() < 0.3
    early = kind == "train" and n <= 400_000 and rng.random() < 0.3
    case = dict(kind=kind, gaussians=n, cameras=cameras, width=width, height=height, scene="city" if city else "box",
                half=600.0 if city else round(half, 1), top=1.0 if city else round(rng.uniform(15.0, 40.0), 1),
                splat=round(rng.uniform(2.0, 5.0), 2) if early else 1.0, geo=not early)
    if kind == "band":
        case["rows"], case["top"] = round(rng.uniform(0.2, 0.9), 3), round(0.13 * case["half"], 1)
    return case


# ----------------------------------------------------------------------------- inputs
def _cameras(case):
    n, W, H, half = case["cameras"], case["width"], case["height"], case["half"]
    if case["scene"] == "city":                     # steep views from 300 m above, on a grid
        cams = []
        for k in range(n):
            eye = ((k % 4 - 0.5) * 300.0, (k // 4 - 0.5) * 300.0, 300.0)
            cams.append(S.look_at_camera(k, eye, (eye[0], eye[1] + 300.0 / math.tan(math.radians(80.0)), 0.0), W, H))
        return cams
    return S.ring_cameras(n, half * 2.0 / 3.0, half * 0.4 + 5.0, W, H)


def _scene(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    with torch.device("cuda"):
        g = S.make_gaussians(case["gaussians"], (case["half"], case["top"]), gen, clustered=case["scene"] == "city")
    if case["splat"] != 1.0:
        g["scales"] *= case["splat"]
    return g, gen


def _settings(cam, geo, bg):
    return GaussianRasterizationSettings(
        image_height=cam.H, image_width=cam.W, tanfovx=cam.tanfovx, tanfovy=cam.tanfovy, bg=bg, scale_modifier=1.0,
        viewmatrix=cam.viewmatrix.cuda(), projmatrix=cam.projmatrix.cuda(), sh_degree=3, campos=cam.campos.cuda(),
        prefiltered=False, render_geo=geo, debug=False)


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device="cuda")


def _leaf(t):
    return t.detach().requires_grad_(True)


def _prepare_raster(case, seed):
    g, gen = _scene(case, seed)
    cams = [c.to("cuda") for c in _cameras(case)]
    geo, train = case["geo"], case["kind"] == "train"
    bg = torch.rand(3, generator=gen, device="cuda") if case["kind"] == "eval" else torch.zeros(3, device="cuda")
    s = dict(kind=case["kind"], settings=[_settings(c, geo, bg) for c in cams], args=make_cuda_args(), geo=geo,
             params={k: _leaf(g[k]) if train else g[k] for k in ("means3D", "scales", "rotations", "opacities")},
             no_sh=torch.empty(0, device="cuda"),
             rgb=[_leaf(S.colours_for(g, c)) if train else S.colours_for(g, c) for c in cams],
             local=torch.ones((case["height"] + 15) // 16, (case["width"] + 15) // 16, dtype=torch.bool,
                              device="cuda"))
    H, W = case["height"], case["width"]
    if train:
        s["flat"] = None if geo else torch.zeros(case["gaussians"], 5, device="cuda")
        s["cot"] = [[_randn(gen, n, H, W) for n in ((3, 5, 1) if geo else (3,))] for _ in cams]
    return s


def _received(case):
    """Records of a band: a little below the share of such a scene that meets a camera's middle `rows`."""
    return max(16, int(0.38 * case["gaussians"] * case["rows"] ** 1.5))


def _prepare_band(case, seed):
    """The records a rank has received for its tile rows of one camera: those whose tiles meet the band."""
    g, gen = _scene(case, seed)
    cam = _cameras(case)[0].to("cuda")
    rs = _settings(cam, case["geo"], torch.zeros(3, device="cuda"))
    H, W = case["height"], case["width"]
    TX, TY = (W + 15) // 16, (H + 15) // 16
    n = max(1, round(TY * case["rows"]))
    row0 = (TY - n) // 2
    with torch.no_grad():
        m2, _, co, radii, depths = GaussianRasterizer(rs).preprocess_gaussians(
            g["means3D"], g["scales"], g["rotations"], torch.empty(0, device="cuda"), g["opacities"], make_cuda_args())
        am = plane_map(g["means3D"], g["scales"], g["rotations"], rs.viewmatrix, rs.campos, radii)
        r = radii.float()
        meets = (radii > 0) & (m2[:, 0] + r > 0) & (m2[:, 0] - r < W) & (m2[:, 1] + r > row0 * 16) & \
            (m2[:, 1] - r < (row0 + n) * 16)
        keep = torch.argsort((~meets).byte(), stable=True)[:_received(case)]
        rgb = S.colours_for(g, cam)
    local = torch.zeros(TY, TX, dtype=torch.bool, device="cuda")
    local[row0:row0 + n] = True
    return dict(kind="band", settings=[rs], args=make_cuda_args(), local=local, radii=radii[keep].contiguous(),
                depths=depths[keep].contiguous(), m2=_leaf(m2[keep]), co=_leaf(co[keep]), rgb=_leaf(rgb[keep]),
                all_map=_leaf(am[keep]), cot=[_randn(gen, 3, H, W), _randn(gen, 5, H, W), _randn(gen, 1, H, W)])


def _prepare_step(case, seed):
    g, _ = _scene(case, seed)
    step = TrainingStep({k: v.cpu() for k, v in g.items()}, _cameras(case), torch.device("cuda"), seed=seed)
    step.enable_densification_stats()
    return dict(kind="step", step=step)


def _prepare_filter(case, seed):
    g, _ = _scene(case, seed)
    bg = torch.zeros(3, device="cuda")
    return dict(kind="filter", settings=[_settings(c, True, bg) for c in _cameras(case)], g=g)


def _prepare_loss(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    H, W = case["height"], case["width"]
    gt = torch.rand(3, (H + 7) // 8, (W + 7) // 8, generator=gen, device="cuda")
    gt = torch.nn.functional.interpolate(gt[None], size=(H, W), mode="bilinear")[0].contiguous()
    image = (gt + 0.1 * _randn(gen, 3, H, W)).clamp(0, 1)       # a render that resembles its photograph
    yy, xx = torch.meshgrid(torch.arange(H, device="cuda"), torch.arange(W, device="cuda"), indexing="ij")
    depth = 100.0 + 0.01 * xx + 0.02 * yy + 0.5 * torch.rand(H, W, generator=gen, device="cuda")
    mask = None
    if case["mask"]:                                            # moving objects cut out in blocks
        keep = torch.rand(1, 1, (H + 31) // 32, (W + 31) // 32, generator=gen, device="cuda") > 0.1
        mask = torch.nn.functional.interpolate(keep.float(), scale_factor=32)[0, 0, :H, :W] > 0.5
    return dict(kind="loss", image=_leaf(image), gt=gt, mask=mask, depth=_leaf(depth), k=(0.8 * W, 0.8 * W, W / 2, H / 2),
                cot=_randn(gen, 3, H, W))


def _prepare_stats(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, off = case["anchors"], case["offsets"]
    seen = torch.rand(n, generator=gen, device="cuda") < case["seen"]
    slots = int(seen.sum()) * off
    selected = torch.rand(slots, generator=gen, device="cuda") < case["selected"]
    gaussians = int(selected.sum())
    return dict(kind="stats", stats=AnchorStatistics(n, off, torch.device("cuda")), seen=seen, selected=selected,
                grad=_randn(gen, gaussians, 2), opacity=torch.tanh(_randn(gen, slots, 1)),
                on_screen=torch.rand(gaussians, generator=gen, device="cuda") < 0.8)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("train", "eval"):
        return _prepare_raster(case, seed)
    return dict(band=_prepare_band, step=_prepare_step, filter=_prepare_filter, loss=_prepare_loss,
                stats=_prepare_stats)[kind](case, seed)


# ----------------------------------------------------------------------------- one pass
def _train(s):
    p = s["params"]
    for t in list(p.values()) + s["rgb"]:
        t.grad = None
    screen = preprocess_gaussians_batched(p["means3D"], p["scales"], p["rotations"], s["no_sh"], p["opacities"],
                                          s["settings"], s["args"], planes=s["geo"])
    heads, cots, out = [], [], []
    for k, rs in enumerate(s["settings"]):
        means2D, _, conic_opacity, radii, depths = screen[k][:5]
        means2D.retain_grad()                                   # the densifier reads it
        means2D_abs = torch.zeros(means2D.shape[0], 3, device="cuda", requires_grad=True)
        color, _, _, _, observe, all_map, depth = GaussianRasterizer(rs).render_gaussians(
            means2D, means2D_abs, conic_opacity, s["rgb"][k], screen[k][5] if s["geo"] else s["flat"], depths, radii,
            s["local"], None, s["args"])
        heads += [color, all_map, depth] if s["geo"] else [color]
        cots += s["cot"][k]
        out.append([color, all_map, depth, observe, means2D, means2D_abs])
    torch.autograd.backward(heads, cots)
    return dict(cameras=[[c.detach(), m.detach(), d.detach(), o, m2.grad, m2a.grad, rgb.grad]
                         for (c, m, d, o, m2, m2a), rgb in zip(out, s["rgb"])],
                grads=[t.grad for t in p.values()])


def _band(s):
    leaves = (s["m2"], s["co"], s["rgb"], s["all_map"])
    for t in leaves:
        t.grad = None
    m2abs = torch.zeros(s["m2"].shape[0], 3, device="cuda", requires_grad=True)
    color, n_render, n_consider, n_contrib, observe, all_map, depth = GaussianRasterizer(s["settings"][0]) \
        .render_gaussians(s["m2"], m2abs, s["co"], s["rgb"], s["all_map"], s["depths"], s["radii"], s["local"], None,
                          s["args"])
    torch.autograd.backward([color, all_map, depth], s["cot"])
    return [color.detach(), all_map.detach(), depth.detach(), n_render, n_consider, n_contrib, observe, m2abs.grad] + \
        [t.grad for t in leaves]


def _eval(s):
    p, rs = s["params"], s["settings"][0]
    rast = GaussianRasterizer(rs)
    with torch.no_grad():
        m2, _, co, radii, depths = rast.preprocess_gaussians(p["means3D"], p["scales"], p["rotations"], s["no_sh"],
                                                             p["opacities"], s["args"])
        am = plane_map(p["means3D"], p["scales"], p["rotations"], rs.viewmatrix, rs.campos, radii)
        color, n_render, n_consider, n_contrib, observe, all_map, depth = rast.render_gaussians(
            m2, None, co, s["rgb"][0], am, depths, radii, s["local"], None, s["args"])
    return [color, all_map, depth, radii, n_render, n_consider, n_contrib, observe]


def _step(s):
    step = s["step"]
    params = step.run()
    d = step.densify
    return dict(grads=[t.grad for t in params.values()], screen=[[r, m.grad] for r, m in step.last],
                stats=[d.grad_accum, d.denom, d.max_radii2D])


def _filter(s):
    g = s["g"]
    return [GaussianRasterizer(rs).visible_filter(g["means3D"], g["scales"], g["rotations"]) for rs in s["settings"]]


def _loss(s):
    image, depth = s["image"], s["depth"]
    image.grad = depth.grad = None
    l1, ssim = strip_loss_sums(image, s["gt"], s["mask"])
    n = float(image.numel())
    loss = 0.8 * (l1 / n) + 0.2 * (1.0 - ssim / n)
    normal = depth_normal(depth, *s["k"])
    torch.autograd.backward([loss, normal], [None, s["cot"]])
    return [l1.detach(), ssim.detach(), image.grad, normal.detach(), depth.grad]


def _stats(s):
    a = s["stats"]
    a.training_statis(s["grad"], s["opacity"], s["on_screen"], s["selected"], s["seen"])
    return [a.opacity_accum, a.anchor_demon, a.offset_gradient_accum, a.offset_denom]


_RUN = dict(train=_train, band=_band, eval=_eval, step=_step, filter=_filter, loss=_loss, stats=_stats)


def run(state):
    return _RUN[state["kind"]](state)


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "stats":
        n, off = case["anchors"], case["offsets"]
        slots = n * case["seen"] * off
        g = slots * case["selected"]
        # masks, opacities and gradients in; the four accumulators in and out (the slots' ones where they change)
        return {"bytes": n + slots * 5 + g * 9 + 16 * n * case["seen"] + 16 * g, "flops": 4 * slots + 6 * g}
    px = case["width"] * case["height"]
    if kind == "loss":
        # image, photograph, mask, depth, cotangent in; gradients and normals out; five 11 + 11-tap window sums each way
        return {"bytes": px * (12 + 12 + bool(case["mask"]) + 4 + 12 + 12 + 12 + 4),
                "flops": px * (3 * (2 * 5 * 22 + 40) + 3 * (2 * 3 * 22 + 20) + 150)}
    P, B = case["gaussians"], case["cameras"]
    if kind == "filter":
        return {"bytes": 40 * P + 4 * P * B, "flops": P * B * 150}
    maps = 9 if case["geo"] else 3
    if kind == "eval":
        return {"bytes": 44 * P + 12 * P + 8 * P + 36 * px, "flops": 250 * P + px * 15 * 40}
    if kind == "band":
        P, px = _received(case), px * case["rows"]
        return {"bytes": P * (8 + 16 + 12 + 20 + 8) + P * (4 + 8 + 12 + 16 + 12 + 20) + 72 * px,
                "flops": px * 15 * 160}
    # parameters and colours in, their gradients and the screen-space ones out; images out, their cotangents in
    return {"bytes": P * 88 + P * B * (12 + 12 + 4 + 8 + 12) + px * B * (36 + 4 * maps),
            "flops": P * B * 600 + px * B * 15 * 160}


def tolerance(case):
    """Images and integers come from the same 32-bit operations whatever the split of the work; the gradients are
    32-bit sums in an order of their own, behind quotients by (1 - alpha) and by the blended normal's projection on
    the ray, which is near zero in places."""
    if case["kind"] == "filter":
        return "exact"
    if case["kind"] in ("loss", "stats"):
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 1e-4, "max": 1e-2}
