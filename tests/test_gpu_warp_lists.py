"""Each warp of the blend kernels feeds itself 32 entries at a time in three stages: lists that end before, at and after a batch, warps whose pixels finish early or
hang over the image, on both sides of the tile counts at which a thread owns two pixels (four tiles per SM backward, eight forward), against the oracle."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(DEV)


@pytest.mark.parametrize("W,H", [(41, 23), (490, 331), (640, 480)])       # 6, 651 and 1,200 tiles
@pytest.mark.parametrize("n,opacity", [(1, 0.0), (31, -2.0), (32, -2.0), (33, -2.0), (64, -3.0), (65, 1.0), (97, -3.0), (130, 3.0)])
def test_list_lengths(pkg, orc, synth, W, H, n, opacity):
    rng = np.random.default_rng(n)
    # every Gaussian covers the image, so every list holds all of them; the last entries, small ones, a corner only
    scale = np.where(np.arange(n) % 8 == 7, -3.0, 0.3)
    P = dict(means=0.2 * rng.standard_normal((n, 3)), sh0=0.5 * rng.standard_normal((n, 1, 3)), shN=np.zeros((n, 0, 3)),
             scaling_raw=scale[:, None] + 0.2 * rng.standard_normal((n, 3)), rotation_raw=rng.standard_normal((n, 4)),
             opacity_raw=opacity + rng.standard_normal((n, 1)))
    P = {k: np.ascontiguousarray(v, np.float32) for k, v in P.items()}
    vm, K = synth.hemisphere_poses(1, 4.0)[0], synth.intrinsics(1.2 * W, 1.2 * W, W / 2.0, H / 2.0)
    bg = np.array([0.2, 0.4, 0.1], np.float32)
    fwd = orc.render_fwd(P, vm, K, W, H, 0, background=bg)
    assert np.diff(np.append(fwd["tile_offsets"].reshape(-1), fwd["flatten_ids"].size)).max() >= n - n // 8
    tr = pkg.trainer
    model = tr.SplatData(n, 1, DEV).load(P)
    grads, rast = model.like(), tr.Rasterizer(model, W, H, 0)
    out = rast.forward(tr.Camera(T(vm), T(K), W, H), T(bg))
    # a pair at the 1/255 cut moves its pixel by 4e-3 of a colour at most
    diff = np.abs(out.image.cpu().numpy() - fwd["render"]).max(-1)
    assert diff.max() < 1e-2 and (diff > 1e-4).sum() <= W * H // 500, (diff.max(), (diff > 1e-4).sum())
    v = rng.normal(size=(H, W, 3)).astype(np.float32) * 1e-3
    bwd = orc.render_bwd(P, fwd, vm, K, W, H, 0, v, background=bg)
    rast.backward(T(v), grads, T(bg))
    for name in ("means", "sh0", "scaling_raw", "rotation_raw", "opacity_raw"):
        # random output gradients cancel over the pixels of a Gaussian: a pair on the other side of the cut weighs a thousandth
        assert rel_l2(grads.tensor(name).cpu().numpy(), bwd[name]) < 2e-3, name
