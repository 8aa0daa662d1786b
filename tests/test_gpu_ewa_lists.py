"""Each warp of the EWA blend kernels walks its own list in batches of 32: lists that end before, at and after a batch and warps that finish early or hang over
the image, on both sides of the tile counts at which a thread owns two pixels (four tiles per SM backward, sixteen forward), against the oracle."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(DEV)


@pytest.mark.parametrize("W,H", [(41, 23), (500, 340), (1030, 600)])       # 6, 704 and 2,470 tiles
@pytest.mark.parametrize("n,opacity", [(1, 0.0), (31, -2.0), (32, -2.0), (33, -2.0), (65, 1.0), (130, 3.0)])
def test_list_lengths(pkg, orc, synth, W, H, n, opacity):
    rng = np.random.default_rng(n)
    scale = np.where(np.arange(n) % 8 == 7, -3.0, 0.3)
    P = dict(means=0.2 * rng.standard_normal((n, 3)), sh0=0.5 * rng.standard_normal((n, 1, 3)), shN=np.zeros((n, 0, 3)),
             scaling_raw=scale[:, None] + 0.2 * rng.standard_normal((n, 3)), rotation_raw=rng.standard_normal((n, 4)),
             opacity_raw=opacity + rng.standard_normal((n, 1)))
    P = {k: np.ascontiguousarray(v, np.float32) for k, v in P.items()}
    vm, K = synth.hemisphere_poses(1, 4.0)[0], synth.intrinsics(1.2 * W, 1.2 * W, W / 2.0, H / 2.0)
    bg = np.array([0.2, 0.4, 0.1], np.float32)
    campos = orc.campos(vm)
    fwd = orc.ewa_forward(P, vm, campos, W, H, K[0, 0], K[1, 1], K[0, 2], K[1, 2], 1, background=bg)
    tr = pkg.trainer
    model = tr.SplatData(n, 1, DEV).load(P)
    grads, rast = model.like(), tr.FastRasterizer(model, W, H, 0)
    out = rast.forward(tr.Camera(T(vm), T(K), W, H), T(bg), cam_position=T(np.asarray(campos, np.float32)))
    # a pair at the 1/255 cut moves its pixel by 4e-3 of a colour at most
    diff = np.abs(out.image.cpu().numpy() - fwd["image"]).max(0)
    assert diff.max() < 1e-2 and (diff > 1e-4).sum() <= W * H // 500, (diff.max(), (diff > 1e-4).sum())
    v = rng.normal(size=(3, H, W)).astype(np.float32) * 1e-3
    bwd = orc.ewa_backward(P, fwd, v)
    rast.backward(T(v), grads, T(bg))
    for name in ("means", "sh0", "scaling_raw", "rotation_raw", "opacity_raw"):
        # random output gradients cancel over the pixels of a Gaussian: a pair on the other side of the cut weighs a thousandth
        assert rel_l2(grads.tensor(name).cpu().numpy(), bwd[name]) < 2e-3, name
