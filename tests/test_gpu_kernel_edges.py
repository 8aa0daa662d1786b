"""Sizes at which the kernels change path or leave a remainder: lists counted and filled by one or by several warps per 32 Gaussians, grids on both sides
of the two-pixel rules, camera boxes under strong distortion, and the row stores of tensors that are not 16-byte aligned."""
import numpy as np
import pytest
import torch

from conftest import make_scene, rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NAMES = ("means", "sh0", "shN", "scaling_raw", "rotation_raw", "opacity_raw")


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


# n: a part of a warp, of a CTA of 256, and more; at and above the 75,776 Gaussians up to which several warps share 32 of them (148 SMs); millions of
# them; radius: rectangles of one tile to 15 x 15
@pytest.mark.parametrize("n,tw,th,rad", [(1, 3, 2, 8.0), (255, 5, 4, 20.0), (256, 5, 4, 20.0), (1025, 40, 3, 40.0), (2047, 9, 7, 24.0),
                                         (2049, 9, 7, 24.0), (70_001, 60, 40, 30.0), (2_097_152, 200, 150, 4.0),
                                         (2_097_153, 200, 150, 4.0), (45_001, 60, 50, 120.0), (75_776, 60, 40, 30.0), (75_777, 60, 40, 30.0)])
def test_tile_lists_against_a_stable_sort(pkg, n, tw, th, rad):
    gen = torch.Generator(device=DEV).manual_seed(n)
    u = lambda *s: torch.rand(s, generator=gen, device=DEV)
    W, H = tw * 16, th * 16
    means2d = torch.stack([u(n) * (W + 40) - 20, u(n) * (H + 40) - 20], -1)[None].contiguous()
    radii = torch.full((1, n, 2), int(rad), dtype=torch.int32, device=DEV)
    radii[0, u(n) < 0.2] = 0
    depths = (u(n) * 64).floor().div(8).add(0.25)[None].contiguous()      # many equal depths: ties go by index
    tiles, ids, flat = pkg.ops.intersect_tile(means2d, radii, depths, None, None, 1, 16, tw, th, True)
    # the same rectangles and order with torch
    m, r = means2d[0] / 16, radii[0].float() / 16
    lo = (m - r).floor().clamp(min=0)
    hi = (m + r).ceil().clamp(min=0)
    size = torch.tensor([tw, th], device=DEV, dtype=torch.float32)
    lo, hi = torch.minimum(lo, size).long(), torch.minimum(hi, size).long()
    w, h = hi[:, 0] - lo[:, 0], hi[:, 1] - lo[:, 1]
    count = torch.where((radii[0] > 0).all(-1), w * h, torch.zeros_like(w))
    assert torch.equal(tiles[0].long(), count)
    g = torch.repeat_interleave(torch.arange(n, device=DEV), count)
    k = torch.arange(g.numel(), device=DEV) - (count.cumsum(0) - count)[g]
    tile = (lo[g, 1] + k // w[g]) * tw + lo[g, 0] + k % w[g]
    key = (tile << 32) | depths[0].view(torch.int32).long()[g]
    order = torch.sort(key, stable=True).indices
    assert flat.numel() == g.numel()
    assert torch.equal(ids, key[order]) and torch.equal(flat.long(), g[order])


# On a 148-SM GPU 37 x 16 tiles are four per SM, the first size of the two-pixel backward, 37 x 32 eight, the first of the two-pixel forward; one column
# fewer stays below
@pytest.mark.parametrize("W,H,lens,mode", [(592, 512, False, 0), (576, 512, False, 0), (601, 523, True, 0), (601, 523, False, 4), (592, 256, False, 0),
                                           (576, 256, False, 0), (592, 256, True, 4), (576, 256, True, 4)])
def test_backward_on_both_sides_of_the_two_pixel_rule(pkg, orc, synth, W, H, lens, mode):
    tr = pkg.trainer
    n, deg = 6000, 1
    cfg, P, vm, K = make_scene(synth, n, W, H, deg, seed=W, fx=500.0)
    radial, tangential = np.array([-0.12, 0.03, 0.0, 0.0, 0.0, 0.0], np.float32), np.array([1e-3, -5e-4], np.float32)
    dist = orc.pack_distortion(radial=radial, tangential=tangential, thin_prism=None) if lens else None
    CH = 3 if mode == 0 else 4
    bg = np.array([0.2, 0.4, 0.1, 0.0], np.float32)[:CH]
    fwd = orc.render_fwd(P, vm, K, W, H, deg, background=bg, radial=dist, render_mode=mode)
    model = tr.SplatData(n, (deg + 1) ** 2, DEV).load(P)
    grads = model.like()
    rast = tr.Rasterizer(model, W, H, deg, render_mode=mode)
    cam = tr.Camera(T(vm), T(K), W, H, **(dict(radial=T(radial), tangential=T(tangential)) if lens else {}))
    out = rast.forward(cam, T(bg))
    # a pair at the 1/255 cut moves its pixel by 4e-3 of a colour at most
    diff = np.abs(out.render.cpu().numpy() - fwd["render"])[..., :3].max(-1)
    assert diff.max() < 1e-2 and (diff > 1e-4).sum() <= W * H // 500, (diff.max(), (diff > 1e-4).sum())
    rng = np.random.default_rng(1)
    v_r = rng.normal(size=(H, W, CH)).astype(np.float32) * 1e-3
    if CH == 4:
        v_r[..., -1] /= float(fwd["depths"][fwd["masks"]].max())
    v_a = rng.normal(size=(H, W, 1)).astype(np.float32) * 1e-3
    bwd = orc.render_bwd(P, fwd, vm, K, W, H, deg, v_r, v_a, background=bg, **(dict(radial=dist) if lens else {}))
    rast.backward(T(v_r), grads, T(bg), T(v_a))
    # a pair whose alpha lies within float32 rounding of the 1/255 cut is blended on one side only and carries its pixel's random
    # output gradient into one Gaussian: two such pairs of 6,000 Gaussians with some 500 pixels each reach 1e-3 on a single tensor
    for name in NAMES:
        assert rel_l2(grads.tensor(name).cpu().numpy(), bwd[name]) < 2e-3, name


# four tiles per SM backward, sixteen (37 x 64) forward
@pytest.mark.parametrize("W,H", [(592, 512), (576, 512), (592, 256), (576, 256), (592, 1024), (576, 1024)])
def test_ewa_backward_on_both_sides_of_the_two_pixel_rule(pkg, orc, synth, W, H):
    tr = pkg.trainer
    n, deg = 6000, 1
    cfg, P, vm, K = make_scene(synth, n, W, H, deg, seed=W, fx=500.0)
    bg = np.array([0.1, 0.2, 0.3], np.float32)
    campos = orc.campos(vm)
    fwd = orc.ewa_forward(P, vm, campos, W, H, K[0, 0], K[1, 1], K[0, 2], K[1, 2], 4, background=bg)
    model = tr.SplatData(n, 4, DEV).load(P)
    rast, grads = tr.FastRasterizer(model, W, H, deg), model.like()
    out = rast.forward(tr.Camera(T(vm), T(K), W, H), T(bg), cam_position=T(np.asarray(campos, np.float32)))
    diff = np.abs(out.image.cpu().numpy() - fwd["image"]).max(0)
    assert diff.max() < 1e-2 and (diff > 1e-4).sum() <= W * H // 500, (diff.max(), (diff > 1e-4).sum())
    gi = np.random.default_rng(2).normal(size=(3, H, W)).astype(np.float32) * 1e-3
    bwd = orc.ewa_backward(P, fwd, gi)
    rast.backward(T(gi), grads, T(bg))
    for name in NAMES:
        assert rel_l2(grads.tensor(name).cpu().numpy(), bwd[name]) < 1e-3, name


# Large and near Gaussians under wide and strongly distorted lenses: a box that is too small drops pairs, which shows as an error of
# the size of an alpha (pairs at the 1/255 cut: 4e-3 of a colour at most, in the few pixels that have one)
@pytest.mark.parametrize("fisheye,coeffs,fx,dist,grow", [
    (True, [0.0, 0.0, 0.0, 0.0], 45.0, 1.6, 1.2), (True, [-0.05, 0.02, -0.004, 0.0], 45.0, 1.1, 0.5),
    (True, [0.03, -0.01, 0.002, 0.001], 60.0, 2.5, 0.0), (False, [-0.3, 0.12, -0.02, 0.01, 0.0, 0.0], 90.0, 1.5, 0.8),
    (False, [0.25, 0.05, 0.0, 0.0, 0.02, 0.0], 120.0, 2.2, 0.3)])
def test_boxes_of_wide_and_distorted_lenses_lose_nothing(pkg, orc, synth, fisheye, coeffs, fx, dist, grow):
    tr, capi = pkg.trainer, pkg._capi
    n, W, H, deg = 3000, 180, 140, 1
    P = synth.make_gaussians(n, 3, "cube", deg)
    P["scaling_raw"] = (P["scaling_raw"] + np.float32(grow)).astype(np.float32)
    vm = synth.look_at_origin([0.3, -dist, 0.4])
    K = synth.intrinsics(fx, fx * 0.97, W / 2 + 5.0, H / 2 - 3.0)
    radial = np.array(coeffs, np.float32)
    kw = dict(camera_model=orc.FISHEYE, radial=radial) if fisheye else dict(radial=orc.pack_distortion(radial=radial))
    fwd = orc.render_fwd(P, vm, K, W, H, deg, **kw)
    model = tr.SplatData(n, (deg + 1) ** 2, DEV).load(P)
    rast = tr.Rasterizer(model, W, H, deg, camera_model=capi.FISHEYE if fisheye else capi.PINHOLE)
    out = rast.forward(tr.Camera(T(vm), T(K), W, H, capi.FISHEYE if fisheye else capi.PINHOLE, radial=T(radial)), None)
    diff = np.abs(out.image.cpu().numpy() - fwd["render"]).max(-1)
    assert diff.max() < 1e-2 and (diff > 1e-4).sum() <= W * H // 500, (diff.max(), (diff > 1e-4).sum())


@pytest.mark.parametrize("H,W", [(1, 1), (11, 33), (32, 32), (31, 65), (43, 34), (97, 96)])
def test_ssim_tile_edges(pkg, orc, H, W):
    rng = np.random.default_rng(H * 100 + W)
    a, b = rng.random((1, 3, H, W)).astype(np.float32), rng.random((1, 3, H, W)).astype(np.float32)
    ref = orc.fusedssim(a[0], b[0])
    out = pkg.ops.fusedssim(0.01 ** 2, 0.03 ** 2, T(a), T(b), True)
    for k in range(4):
        r = np.asarray(ref[k]).reshape(-1)
        # float32 window sums of values up to 1: 121 roundings of 6e-8, divided by variances of 0.08 and more
        assert np.abs(out[k].cpu().numpy().reshape(-1) - r).max() < 2e-5 * max(1.0, np.abs(r).max()), k
    dl = rng.normal(size=(1, 3, H, W)).astype(np.float32)
    g = pkg.ops.fusedssim_backward(0.01 ** 2, 0.03 ** 2, T(a), T(b), T(dl), *out[1:])
    assert rel_l2(g.cpu().numpy(), orc.fusedssim_backward(a[0], b[0], dl[0], *ref[1:])) < 1e-4


# A model with room for 2,100,000 Gaussians that holds 2,090,000: the workspace is sized for the former and laid out for the latter
@pytest.mark.parametrize("ewa", [False, True])
def test_fewer_gaussians_than_the_workspace_was_made_for(pkg, synth, ewa):
    tr = pkg.trainer
    W, H, n, capacity = 96, 64, 2_090_000, 2_100_000
    _, P, vm, K = make_scene(synth, 1000, W, H, 0)
    model = tr.SplatData(n, 1, DEV, capacity=capacity)
    for name in NAMES:
        t = model.tensor(name)
        if t.numel():
            t.copy_(T(P[name]).repeat(n // 1000, *[1] * (t.dim() - 1)).view(t.shape))
    cam, bg = tr.Camera(T(vm), T(K), W, H), torch.zeros(3, device=DEV)
    make = (lambda m: tr.FastRasterizer(m, W, H, 0, instance_capacity=1 << 25)) if ewa else (lambda m: tr.Rasterizer(m, W, H, 0, isect_capacity=1 << 25))
    image = make(model).forward(cam, bg).image.clone()
    exact = tr.SplatData(n, 1, DEV)
    for name in NAMES:
        exact.tensor(name).copy_(model.tensor(name))
    assert torch.isfinite(image).all() and image.abs().max() > 0.1
    assert torch.equal(image, make(exact).forward(cam, bg).image)


# Keys that belong to no tile, the largest there are: every tile's list is empty
@pytest.mark.parametrize("n,C,tw,th", [(1, 1, 3, 2), (5000, 1, 81, 53), (300, 3, 7, 5)])
def test_offsets_of_a_list_that_was_given_up(pkg, n, C, tw, th):
    ids = torch.full((n,), torch.iinfo(torch.int64).max, dtype=torch.int64, device=DEV)
    assert (pkg.ops.intersect_offset(ids, C, tw, th) == 0).all()


# An equirectangular camera inside the scene, on both sides of the tile counts at which a thread owns two pixels (4 per SM backward, 8 forward): 512, 1,250
# and 2,048 tiles.
@pytest.mark.parametrize("W,H", [(512, 256), (800, 400), (1024, 512)])
def test_equirectangular_on_both_sides_of_the_two_pixel_rules(pkg, orc, synth, W, H):
    tr, capi = pkg.trainer, pkg._capi
    n, deg = 4000, 1
    P = synth.make_gaussians(n, 6, "cube", deg)
    P["scaling_raw"] = (P["scaling_raw"] + np.float32(0.7)).astype(np.float32)
    vm = np.eye(4, dtype=np.float32)
    vm[:3, 3] = [0.05, -0.02, 0.1]
    K, bg = synth.intrinsics(100.0, 100.0, W / 2, H / 2), np.array([0.2, 0.4, 0.1], np.float32)
    fwd = orc.render_fwd(P, vm, K, W, H, deg, background=bg, camera_model=orc.EQUIRECTANGULAR)
    model = tr.SplatData(n, (deg + 1) ** 2, DEV).load(P)
    grads, rast = model.like(), tr.Rasterizer(model, W, H, deg, camera_model=capi.EQUIRECTANGULAR)
    out = rast.forward(tr.Camera(T(vm), T(K), W, H, capi.EQUIRECTANGULAR), T(bg))
    # azimuths and elevations come from single-precision arc functions on both sides: a projection that rounds differently moves a tile of a faint rim
    diff = np.abs(out.image.cpu().numpy() - fwd["render"]).max(-1)
    assert diff.max() < 1e-2 and (diff > 1e-4).sum() <= W * H // 500, (diff.max(), (diff > 1e-4).sum())
    v = np.random.default_rng(1).normal(size=(H, W, 3)).astype(np.float32) * 1e-3
    bwd = orc.render_bwd(P, fwd, vm, K, W, H, deg, v, background=bg, camera_model=orc.EQUIRECTANGULAR)
    rast.backward(T(v), grads, T(bg))
    for name in NAMES:
        assert rel_l2(grads.tensor(name).cpu().numpy(), bwd[name]) < 2e-3, name
