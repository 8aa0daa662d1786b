"""The work that users of this framework have it do, as cases that can be timed one by one.

A case is a dict of plain values; its "path" says which public entry points it goes through:

  step   one training step of the gsplat / 3DGUT path on one GPU: Rasterizer.forward, PhotometricLoss,
         Rasterizer.backward and the fused Adam. With one camera the shN gradient is used in its rank-1 form
         (backward(write_shN=False) + adam_step_rank1_sh), with more cameras the gradients accumulate and
         adam_step_splats runs once
  mcmc   the same step driven by the MCMC strategy in its own order: backward, regularisers, post_backward (noise
         injection; the iteration is not a refining one), strategy.step
  ewa    one training step of the default EWA path: FastRasterizer.forward / backward with densification statistics
  render a forward-only render, as for evaluation or a preview
  ops    the operator-level pair rasterize_from_world_with_sh_fwd / _bwd of a host program that keeps its own autograd

Scenes have the value distributions of the synthetic configurations (clusters, wide, cube) and are drawn on the GPU;
where a clustered scene has fewer than a million Gaussians they are larger in proportion, as a coarser model is.
Learning rates are a hundredth of the configured ones, the end of the exponential schedule, and the Adam moments are
those of a run under way, so that a scene stays the one the case describes however often the step is repeated."""
from __future__ import annotations

import importlib
import math

import torch

lfs = importlib.import_module("lichtfeld-studio_b200")
synth, tr, strategy, ops, capi = lfs.synth, lfs.trainer, lfs.strategy, lfs.ops, lfs._capi

LRS = [1.6e-6, 2.5e-5, 1.25e-6, 5e-5, 1e-5, 5e-4]   # means, sh0, shN, scaling, rotation, opacity
CAMERAS = {"pinhole": capi.PINHOLE, "opencv": capi.PINHOLE, "fisheye": capi.FISHEYE}
MODES = {"rgb": tr.RENDER_RGB, "rgb_ed": tr.RENDER_RGB_ED}
TRAINED = ("means", "sh0", "scaling_raw", "rotation_raw", "opacity_raw")


def _case(name, path, n, W, H, **kw):
    c = dict(path=path, n=n, W=W, H=H, layout="clusters", sh_coeffs=16, degree=3, camera="pinhole", cameras=1, antialiased=False,
             mode="rgb")
    if name is not None:
        c["name"] = name
    c.update(kw)
    return c


def listed():
    return [
        # the smallest step: an object-sized scene without view dependence, where launches and host time count
        _case("step_16k_256", "step", 16_384, 256, 256, layout="cube", sh_coeffs=1, degree=0),
        # the first minutes of a run: a structure-from-motion start, SH degree 1 of 3 active, images at a reduced, odd size
        _case("mcmc_120k_979x547", "mcmc", 120_003, 979, 547, degree=1),
        # a distorted-lens capture, the reason to train with the unscented transform, with the antialiased option
        _case("step_opencv_400k_1237x823", "step", 400_000, 1237, 823, camera="opencv", antialiased=True),
        # a 180 degree fisheye capture
        _case("step_fisheye_250k_1024", "step", 250_000, 1024, 1024, camera="fisheye", degree=2),
        # the benchmark's training step
        _case("step_1m_1296x840", "step", 1_000_000, 1296, 840),
        # the large training step: the data-parallel configuration's model and images, two cameras per optimizer step
        _case("step_3m_1600x1064_x2", "step", 3_000_000, 1600, 1064, cameras=2),
        # the default rasterizer's step early in a run and at the benchmark's size
        _case("ewa_60k_777x519", "ewa", 60_001, 777, 519, degree=1),
        _case("ewa_1m_1296x840", "ewa", 1_000_000, 1296, 840),
        # a preview frame with depth
        _case("render_150k_640x360_depth", "render", 150_000, 640, 360, mode="rgb_ed"),
        # large-scene evaluation renders: 4K pinhole and 180 degree fisheye
        _case("render_6m_4k", "render", 6_000_000, 3840, 2160, layout="wide"),
        _case("render_6m_fisheye_1920", "render", 6_000_000, 1920, 1920, layout="wide", camera="fisheye"),
        # the operator pair under a host's own autograd
        _case("ops_250k_640x427", "ops", 250_000, 640, 427),
    ]


def draw(rng):
    path = rng.choice(["step", "step", "step", "mcmc", "ewa", "ewa", "render", "render", "ops"])
    log = lambda lo, hi: int(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    n = log(10_000, 4_000_000 if path == "render" else 1_500_000)
    pixels, aspect = log(60_000, 6_000_000 if path == "render" else 1_500_000), rng.uniform(0.75, 1.9)
    W, H = int(math.sqrt(pixels * aspect)), int(math.sqrt(pixels / aspect))
    kw = dict(degree=rng.choice([0, 1, 2, 3, 3, 3]))
    if path in ("step", "render", "ops"):
        kw["camera"] = rng.choice(["pinhole", "pinhole", "opencv", "fisheye"])
    if path in ("step", "render"):
        kw["antialiased"] = rng.random() < 0.3
    if path == "step":
        kw["cameras"] = rng.choice([1, 1, 1, 2])
    if path == "render":
        kw["layout"] = rng.choice(["clusters", "wide"])
        kw["mode"] = rng.choice(["rgb", "rgb", "rgb_ed"])
    return _case(None, path, n, W, H, **kw)


# ---------------------------------------------------------------------------------------------------------------------
def _scene(case, gen, dev):
    n, K = case["n"], case["sh_coeffs"]
    normal = lambda *s: torch.randn(s, generator=gen, device=dev)
    uniform = lambda *s: torch.rand(s, generator=gen, device=dev)
    if case["layout"] == "cube":
        means, mu, sd, opacity = uniform(n, 3) * 2 - 1, -4.0, 0.5, 0.0
    elif case["layout"] == "clusters":
        centres = uniform(64, 3) * 4.2 - 2.1
        means = (centres[torch.arange(n, device=dev) % 64] + 0.3 * normal(n, 3)).clamp_(-3, 3)
        mu, sd, opacity = -4.5 + max(0.0, math.log(1e6 / n) / 3), 0.6, -1.0
    else:
        means, mu, sd, opacity = uniform(n, 3) * 20 - 10, -5.0, 0.7, -1.0
    return dict(means=means, sh0=0.5 * normal(n, 1, 3), shN=0.05 * normal(n, K - 1, 3), scaling_raw=mu + sd * normal(n, 3),
                rotation_raw=torch.nn.functional.normalize(normal(n, 4), dim=-1), opacity_raw=opacity + normal(n, 1))


def _cameras(case, gen, dev, count):
    """`count` poses of the configuration's hemisphere, intrinsics for the same field of view at any image size."""
    W, H, model = case["W"], case["H"], CAMERAS[case["camera"]]
    if case["layout"] == "cube":
        poses, f = synth.hemisphere_poses(64, 4.0), W * 300.0 / 256.0
    elif case["layout"] == "clusters":
        poses, f = synth.hemisphere_poses(200, 5.0), W * 1150.0 / 1296.0
    else:
        poses, f = synth.hemisphere_poses(32, 12.0), W * 2800.0 / 3840.0
    if model == capi.FISHEYE:
        f = min(W, H) / math.pi   # 180 degrees across the shorter side
    K = torch.from_numpy(synth.intrinsics(f, f, W / 2.0, H / 2.0)).to(dev)
    lens = {}
    if case["camera"] == "opencv":
        lens = dict(radial=torch.tensor([-0.06, 0.012, -0.001, 0.0, 0.0, 0.0], device=dev),
                    tangential=torch.tensor([4e-4, -3e-4], device=dev), thin_prism=torch.tensor([1e-4, 0.0, -1e-4, 0.0], device=dev))
    elif model == capi.FISHEYE:
        lens = dict(radial=torch.zeros(4, device=dev))
    pick = torch.randperm(len(poses), generator=gen, device=dev)[:count].tolist()
    return [tr.Camera(torch.from_numpy(poses[i]).to(dev), K, W, H, model, **lens) for i in pick]


def _photos(case, gen, dev, count):
    """Target images with broad structure and some grain."""
    H, W, out = case["H"], case["W"], []
    for _ in range(count):
        broad = torch.rand((1, 3, 12, 16), generator=gen, device=dev)
        img = torch.nn.functional.interpolate(broad, size=(H, W), mode="bilinear", align_corners=False)[0]
        out.append((img + 0.05 * torch.randn((3, H, W), generator=gen, device=dev)).clamp_(0, 1).contiguous())
    return out


def _moments(model, gen, pixels):
    """Adam moments of the size that gradients of a mean over `pixels` have."""
    m, v = model.like(), model.like()
    m.flat.normal_(generator=gen).mul_(0.3 / pixels)
    v.flat.normal_(generator=gen).mul_(0.5 / pixels).square_().add_((0.5 / pixels) ** 2)
    return m, v


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    n, K, W, H, path = case["n"], case["sh_coeffs"], case["W"], case["H"], case["path"]
    scene = _scene(case, gen, dev)
    cams = _cameras(case, gen, dev, case["cameras"])
    s = dict(case=case, cams=cams, background=torch.rand(3, generator=gen, device=dev), step=1000)
    if path == "ops":
        s["args"] = (scene["means"], scene["rotation_raw"], scene["scaling_raw"].exp(), scene["opacity_raw"].sigmoid().squeeze(-1),
                     torch.cat([scene["sh0"], scene["shN"]], 1))
        s["v_render"] = torch.randn((1, H, W, 3), generator=gen, device=dev) / (3 * H * W)
        s["v_alpha"] = torch.zeros((1, H, W, 1), device=dev)
        return s
    model = s["model"] = tr.SplatData(n, K, dev).load(scene)
    capacity = max(24 * n, 1 << 22)
    if path == "ewa":
        s["rasterizer"] = tr.FastRasterizer(model, W, H, case["degree"], instance_capacity=capacity)
        s["densification"] = torch.zeros((2, n), device=dev)
        s["hwc"], s["chw"] = torch.empty((H, W, 3), device=dev), torch.empty((3, H, W), device=dev)
    else:
        s["rasterizer"] = tr.Rasterizer(model, W, H, case["degree"], cams[0].camera_model, isect_capacity=capacity,
                                        render_mode=MODES[case["mode"]], antialiased=case["antialiased"])
    if path == "render":
        return s
    s["photos"] = _photos(case, gen, dev, case["cameras"])
    s["loss"] = tr.PhotometricLoss(W, H, dev)
    if path == "mcmc":
        st = s["strategy"] = strategy.MCMC(model)
        st.initialize(strategy.OptimizationParameters(means_lr=LRS[0], shs_lr=LRS[1], scaling_lr=LRS[3], rotation_lr=LRS[4],
                                                      opacity_lr=LRS[5], max_cap=n))
        st._optimizer.exp_avg, st._optimizer.exp_avg_sq = _moments(model, gen, H * W)
        torch.manual_seed(seed)   # the injected noise comes from torch's own generator
        return s
    s["grads"] = model.like()
    s["exp_avg"], s["exp_avg_sq"] = _moments(model, gen, H * W)
    return s


def _learned(model, exp_avg, exp_avg_sq, grads, loss):
    return {"loss": loss[:1], "model": model.flat, "exp_avg": exp_avg.flat, "exp_avg_sq": exp_avg_sq.flat,
            "grads": {k: grads.tensor(k) for k in TRAINED}}


def _run_step(s):
    rast, grads, bg = s["rasterizer"], s["grads"], s["background"]
    s["step"] += 1
    several = len(s["cams"]) > 1
    for c, (cam, photo) in enumerate(zip(s["cams"], s["photos"])):
        out = rast.forward(cam, bg)
        loss, v_render = s["loss"](out.image, photo)
        rast.backward(v_render, grads, bg, accumulate=c > 0, write_shN=several)
    if several:
        tr.adam_step_splats(s["model"], s["exp_avg"], s["exp_avg_sq"], grads, LRS, s["step"], grad_scale=1.0 / len(s["cams"]))
    else:
        rast.adam_step_rank1_sh(s["exp_avg"], s["exp_avg_sq"], grads, LRS, s["step"])
    got = _learned(s["model"], s["exp_avg"], s["exp_avg_sq"], grads, loss)
    got.update(image=out.image, alpha=out.alpha, overflow=out.status[:1])
    if several:
        got["grads"]["shN"] = grads.tensor("shN")
    return got


def _run_mcmc(s):
    rast, st, bg, it = s["rasterizer"], s["strategy"], s["background"], 750
    out = rast.forward(s["cams"][0], bg)
    loss, v_render = s["loss"](out.image, s["photos"][0])
    rast.backward(v_render, st.grads, bg)
    reg = tr.regularization(s["model"], st.grads, 0.01, 0.01)
    st.post_backward(it, out)
    st.step(it)
    got = _learned(s["model"], st._optimizer.exp_avg, st._optimizer.exp_avg_sq, st.grads, loss)
    got["grads"]["shN"] = st.grads.tensor("shN")
    got.update(image=out.image, alpha=out.alpha, overflow=out.status[:1], regularization=reg)
    return got


def _run_ewa(s):
    rast, grads, bg = s["rasterizer"], s["grads"], s["background"]
    s["step"] += 1
    out = rast.forward(s["cams"][0], bg)
    s["hwc"].copy_(out.image.permute(1, 2, 0))        # the loss reads HWC
    loss, v_hwc = s["loss"](s["hwc"], s["photos"][0])
    s["chw"].copy_(v_hwc.permute(2, 0, 1))
    rast.backward(s["chw"], grads, bg, densification_info=s["densification"], write_shN=False)
    rast.adam_step_rank1_sh(s["exp_avg"], s["exp_avg_sq"], grads, LRS, s["step"])
    got = _learned(s["model"], s["exp_avg"], s["exp_avg_sq"], grads, loss)
    got.update(image=out.image, alpha=out.alpha, overflow=out.status[:1], densification=s["densification"])
    return got


def _run_render(s):
    out = s["rasterizer"].forward(s["cams"][0], s["background"])
    return {"image": out.image, "alpha": out.alpha, "status": out.status, "depth": out.depth}


def _run_ops(s):
    c, cam = s["case"], s["cams"][0]
    means, quats, scales, opacities, sh = s["args"]
    bg = s["background"].view(1, 3)
    lens = tuple(None if t is None else t.view(1, -1) for t in (cam.radial, cam.tangential, cam.thin_prism))
    front = (means, quats, scales, opacities, sh, c["degree"], bg, None, c["W"], c["H"], 16, cam.viewmat.view(1, 4, 4), None,
             cam.K.view(1, 3, 3), cam.camera_model, 0.3, 0.01, 10000.0, 0.0, 1.0, False, 0, None, ops.ShutterType.GLOBAL) + lens
    renders, alphas, radii, means2d, depths, colors, offsets, ids, last_ids, comps = ops.rasterize_from_world_with_sh_fwd(*front)
    grads = ops.rasterize_from_world_with_sh_bwd(*front, alphas, last_ids, offsets, ids, colors, radii, means2d, depths, comps,
                                                 s["v_render"], s["v_alpha"])
    # the list of Gaussian ids has another length in every scene; the offsets into it and the pixels' last positions stand for it
    return {"image": renders, "alpha": alphas, "radii": radii, "offsets": offsets, "last_ids": last_ids, "grads": grads}


def run(state):
    return {"step": _run_step, "mcmc": _run_mcmc, "ewa": _run_ewa, "render": _run_render, "ops": _run_ops}[state["case"]["path"]](state)


# ---------------------------------------------------------------------------------------------------------------------
#: (pixel, Gaussian) pairs that a pixel blends, measured on the listed scenes
BLENDED = {("clusters", False): 100, ("clusters", True): 10, ("cube", False): 20, ("wide", False): 35, ("wide", True): 14}


def work(case):
    """bytes: every input read once, every output written once. flops: per Gaussian about 700 (projection, colour, and the
    same again for the gradient), per blended (pixel, Gaussian) pair 45 forward and 100 more backward, 300 per pixel for the
    loss, 12 per parameter for Adam."""
    n, K, path, cams = case["n"], case["sh_coeffs"], case["path"], case["cameras"]
    row, pixels = 11 + 3 * K, case["W"] * case["H"] * cams
    pairs = BLENDED[case["layout"], case["camera"] == "fisheye"] * pixels
    if path == "render":
        channels = 3 if case["mode"] == "rgb" else 4
        return {"bytes": 4.0 * row * n + 4.0 * (channels + 1) * pixels, "flops": 700.0 * n + 45.0 * pairs}
    flops = 1400.0 * n * cams + 145.0 * pairs
    if path == "ops":
        return {"bytes": 4.0 * (2 * row + 2) * n + 4.0 * (3 + 1 + 1 + 4) * pixels, "flops": flops}
    grads = row if path == "mcmc" or cams > 1 else 14
    return {"bytes": 4.0 * (6 * row + grads) * n + 28.0 * pixels, "flops": flops + 300.0 * pixels + 12.0 * row * n}


def tolerance(case):
    """Four times the difference between this framework built with and without contraction of products and sums into FMAs:
    a pair whose alpha lies within rounding of the 1/255 cut falls on either side of it, and each such pair changes a
    pixel by up to 4e-3 and single gradients by more. The EWA path projects once per Gaussian and has far fewer of them.
    (On the same inputs twice, with the backward's atomic sums in another order: 1e-5, 2e-3.)"""
    if case["path"] == "render":
        return {"rel": 1e-4, "max": 0.025}
    if case["path"] == "ewa":
        return {"rel": 1.5e-4, "max": 0.04}
    return {"rel": 2e-3, "max": 0.8, "differ": 4e-4 if case["path"] == "ops" else 0.0}   # differ: the operators' last_ids
