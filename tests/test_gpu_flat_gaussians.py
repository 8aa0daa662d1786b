"""A Gaussian of no thickness (a scale of 0, or exp of a raw scale that leaves no reciprocal): its response is NaN along every ray, and min(0.999, NaN) blends it
with alpha 0.999 into every pixel of its tiles. Forward and backward have to take the same pairs, or the gradients of the Gaussians in front of it are off by the
factor 1 / (1 - 0.999). Image and the others' gradients against the oracle, on both sides of the two-pixel rules."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
FLAT = [3, 11, 20, 41]


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(DEV)


def scene(synth, W, H):
    n = 60
    rng = np.random.default_rng(W)
    scaling = -1.6 + 0.3 * rng.standard_normal((n, 3))
    scaling[FLAT, [0, 1, 2, 1]] = -100.0
    P = dict(means=0.4 * rng.standard_normal((n, 3)), sh0=0.5 * rng.standard_normal((n, 1, 3)), shN=np.zeros((n, 0, 3)), scaling_raw=scaling,
             rotation_raw=rng.standard_normal((n, 4)), opacity_raw=rng.standard_normal((n, 1)) - 1.0)
    P = {k: np.ascontiguousarray(v, np.float32) for k, v in P.items()}
    return P, synth.hemisphere_poses(1, 4.0)[0], synth.intrinsics(1.2 * W, 1.2 * W, W / 2.0, H / 2.0), rng.normal(size=(H, W, 3)).astype(np.float32) * 1e-3


def check_image(got, want, W, H):
    # a pair at the 1/255 cut moves its pixel by 4e-3 of a colour at most
    diff = np.abs(got - want).max(-1)
    assert diff.max() < 1e-2 and (diff > 1e-4).sum() <= W * H // 500, (diff.max(), (diff > 1e-4).sum())


@pytest.mark.parametrize("W,H,lens", [(41, 23, False), (640, 480, False), (1024, 600, False), (137, 90, True)])     # 6, 1,200, 2,432 and 54 tiles
def test_fused(pkg, orc, synth, W, H, lens):
    P, vm, K, v = scene(synth, W, H)
    bg = np.array([0.2, 0.4, 0.1], np.float32)
    model_kw = dict(camera_model=orc.FISHEYE, radial=np.zeros(4, np.float32)) if lens else {}
    fwd = orc.render_fwd(P, vm, K, W, H, 0, background=bg, **model_kw)
    assert (fwd["radii"][FLAT] > 0).all()
    tr, capi = pkg.trainer, pkg._capi
    kind = capi.FISHEYE if lens else capi.PINHOLE
    model = tr.SplatData(60, 1, DEV).load(P)
    grads, rast = model.like(), tr.Rasterizer(model, W, H, 0, camera_model=kind)
    out = rast.forward(tr.Camera(T(vm), T(K), W, H, kind, radial=T(np.zeros(4)) if lens else None), T(bg))
    check_image(out.image.cpu().numpy(), fwd["render"], W, H)
    bwd = orc.render_bwd(P, fwd, vm, K, W, H, 0, v, background=bg, **model_kw)
    rast.backward(T(v), grads, T(bg))
    others = np.setdiff1d(np.arange(60), FLAT)
    # a T of 1 - 0.9995 has lost 11 of its 24 bits before it is divided by 0.001
    for name in ("means", "sh0", "scaling_raw", "rotation_raw", "opacity_raw"):
        assert rel_l2(grads.tensor(name).cpu().numpy()[others], bwd[name][others]) < 2e-3, name


@pytest.mark.parametrize("W,H", [(41, 23), (1024, 600)])
def test_operators(pkg, orc, synth, W, H):
    P, vm, K, v = scene(synth, W, H)
    bg = np.array([0.2, 0.4, 0.1], np.float32)
    P["scaling_raw"][P["scaling_raw"] == -100.0] = -np.inf      # a scale of exactly 0
    fwd = orc.render_fwd(P, vm, K, W, H, 0, background=bg)
    quats, scales, opac = orc.act_quat(P["rotation_raw"])[0], orc.act_scale(P["scaling_raw"]), orc.act_opacity(P["opacity_raw"])
    assert (scales[FLAT] == 0).any(1).all() and (fwd["radii"][FLAT] > 0).all()
    args = [T(P["means"]), T(quats), T(scales), T(fwd["colors"][None]), T(opac[None]), T(bg[None]), None, W, H, 16, T(vm[None]), None, T(K[None]), 0]
    lists = dict(tile_offsets=torch.from_numpy(fwd["tile_offsets"][None]).to(DEV), flatten_ids=torch.from_numpy(fwd["flatten_ids"]).to(DEV))
    render, alpha, last = pkg.ops.rasterize_to_pixels_from_world_3dgs_fwd(*args, **lists)
    check_image(render.cpu().numpy()[0], fwd["render"], W, H)
    zero = np.zeros((H, W, 1), np.float32)
    want = orc.rasterize_bwd(P["means"], quats, scales, fwd["colors"], opac, bg, W, H, 16, vm, K, fwd["tile_offsets"], fwd["flatten_ids"], fwd["alpha"],
                             fwd["last_ids"], v, zero)
    got = pkg.ops.rasterize_to_pixels_from_world_3dgs_bwd(*args, **lists, render_alphas=alpha, last_ids=last, v_render_colors=T(v[None]),
                                                          v_render_alphas=T(zero[None]))
    others = np.setdiff1d(np.arange(60), FLAT)
    for name, a, b in zip(("means", "quats", "scales", "colors", "opacities"), got, want):
        assert rel_l2(a.cpu().numpy().reshape(b.shape)[others], b[others]) < 2e-3, name
