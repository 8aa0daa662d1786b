"""Threads of the blend kernels that skip an entry go through its sums with an alpha of zero, and zero times an infinite colour is not zero: exactly the pixels
that an infinitely bright Gaussian is blended into may be infinite. Its pixels are found with a finite colour. On both sides of the two-pixel rules."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(DEV)


@pytest.mark.parametrize("ewa", [False, True])
@pytest.mark.parametrize("W,H,lens", [(41, 23, False), (1024, 600, False), (137, 90, True)])     # 6, 2,432 and 54 tiles
def test_only_blended_pixels_are_infinite(pkg, synth, W, H, lens, ewa):
    n, k = 40, 17
    rng = np.random.default_rng(W)
    P = dict(means=0.3 * rng.standard_normal((n, 3)), sh0=0.5 * rng.standard_normal((n, 1, 3)), shN=np.zeros((n, 0, 3)),
             scaling_raw=-2.0 + 0.3 * rng.standard_normal((n, 3)), rotation_raw=rng.standard_normal((n, 4)), opacity_raw=rng.standard_normal((n, 1)))
    P = {name: np.ascontiguousarray(v, np.float32) for name, v in P.items()}
    tr = pkg.trainer
    vm, K = synth.hemisphere_poses(1, 4.0)[0], synth.intrinsics(1.2 * W, 1.2 * W, W / 2.0, H / 2.0)
    fisheye = lens and not ewa
    images = []
    for value in (0.0, 1e9, np.inf):
        P["sh0"][k] = value
        model = tr.SplatData(n, 1, DEV).load(P)
        if ewa:
            rast = tr.FastRasterizer(model, W, H, 0)
            out = rast.forward(tr.Camera(T(vm), T(K), W, H), None)
            images.append(out.image.cpu().numpy())
        else:
            capi = pkg._capi
            kind = capi.FISHEYE if fisheye else capi.PINHOLE
            rast = tr.Rasterizer(model, W, H, 0, camera_model=kind)
            cam = tr.Camera(T(vm), T(K), W, H, kind, radial=T(np.zeros(4))) if fisheye else tr.Camera(T(vm), T(K), W, H)
            images.append(rast.forward(cam, None).image.cpu().numpy().transpose(2, 0, 1))
    dark, bright, infinite = images
    assert np.isfinite(dark).all() and np.isfinite(bright).all()
    blended = np.abs(bright - dark).max(0) > 1.0       # 1e9 times alpha and transmittance, at least 4e-7 of it, against colours of 2
    assert 0 < blended.sum() < blended.size
    assert np.array_equal(~np.isfinite(infinite).all(0), blended)
    assert np.array_equal(infinite[:, ~blended], dark[:, ~blended])


# the colours in a call of their own after the lists (the form of the data-parallel step)
@pytest.mark.parametrize("W,H,mode", [(41, 23, 0), (1024, 600, 0), (137, 90, 4)])
@pytest.mark.parametrize("value", [np.inf, 1e9])
def test_split_forward_is_the_whole_one(pkg, synth, W, H, mode, value):
    n = 40
    rng = np.random.default_rng(W)
    P = dict(means=0.3 * rng.standard_normal((n, 3)), sh0=0.5 * rng.standard_normal((n, 1, 3)), shN=0.1 * rng.standard_normal((n, 3, 3)),
             scaling_raw=-2.0 + 0.3 * rng.standard_normal((n, 3)), rotation_raw=rng.standard_normal((n, 4)), opacity_raw=rng.standard_normal((n, 1)))
    P["sh0"][17] = value
    tr = pkg.trainer
    model = tr.SplatData(n, 4, DEV).load({k: np.ascontiguousarray(v, np.float32) for k, v in P.items()})
    rast = tr.Rasterizer(model, W, H, 1, render_mode=mode)
    cam = tr.Camera(T(synth.hemisphere_poses(1, 4.0)[0]), T(synth.intrinsics(1.2 * W, 1.2 * W, W / 2.0, H / 2.0)), W, H)
    whole = rast.forward(cam, None).render.cpu().numpy()
    assert np.isfinite(whole).any() and not (np.isfinite(whole).all() and np.isinf(value))
    rast.forward_lists(cam)
    split = rast.forward_shade(None).render.cpu().numpy()
    assert np.array_equal(whole, split, equal_nan=True)
