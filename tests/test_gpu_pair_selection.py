"""Which (pixel, Gaussian) pairs are blended. The rasterizer evaluates a pair by three linear forms of the pixel's direction and skips
most pairs by boxes and patches; none of that may change the set of pairs whose alpha reaches 1/255."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def fma32(a, b, c):
    """float32 fma: the product of two floats is exact in float64, the sum is rounded there once and then to float32"""
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


# Every tile holds one Gaussian some four pixels wide. The camera's axes are the world's and the focal length is a power of two, so
# the float32 pixel rays have one value whatever is fused; the quaternions have a float32 norm of exactly 1. What remains is the
# product form |u x g|^2 / |u|^2 itself, emulated below operation by operation.
@pytest.mark.parametrize("f,seed,decided", [(32768.0, 0, 10), (262144.0, 1, 100)])
def test_pairs_at_the_cut_are_those_of_the_product_form(pkg, f, seed, decided):
    W = H = 1024
    tw = W // 16
    n = tw * tw
    rng = np.random.default_rng(seed)
    z = np.float32(f / 200.0)
    ty, tx = np.divmod(np.arange(n), tw)
    px, py = tx * 16 + rng.uniform(2, 14, n), ty * 16 + rng.uniform(2, 14, n)
    means = np.stack([(px - 512.0) / f * z, (py - 512.0) / f * z, np.full(n, z) * rng.uniform(0.9, 1.1, n)], -1).astype(np.float32)
    scales = (rng.uniform(2.5, 6.0, (n, 3)) / f * z).astype(np.float32)
    q = rng.normal(size=(20 * n, 4))
    q = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    w, x, y, z_ = q.T
    quats = q[((x * x + y * y) + z_ * z_) + w * w == 1][:n]
    opac = rng.uniform(0.05, 0.95, n).astype(np.float32)
    w, x, y, z_ = quats.T
    one, two = np.float32(1), np.float32(2)
    R = np.array([[one - two * (y * y + z_ * z_), two * (x * y - w * z_), two * (x * z_ + w * y)],
                  [two * (x * y + w * z_), one - two * (x * x + z_ * z_), two * (y * z_ - w * x)],
                  [two * (x * z_ - w * y), two * (y * z_ + w * x), one - two * (x * x + y * y)]]).transpose(2, 0, 1)
    M = (one / scales)[:, :, None] * R.transpose(0, 2, 1)
    om = -means
    g = M[:, :, 0] * om[:, None, 0] + M[:, :, 1] * om[:, None, 1] + M[:, :, 2] * om[:, None, 2]
    assert len(quats) == n and M.dtype == g.dtype == np.float32
    # pixels of a tile: [n, 256]
    lx, ly = np.arange(256) % 16, np.arange(256) // 16
    ux = ((tx[:, None] * 16 + lx + 0.5 - 512.0) / f).astype(np.float32)
    uy = ((ty[:, None] * 16 + ly + 0.5 - 512.0) / f).astype(np.float32)
    length = np.sqrt((ux * ux + uy * uy) + np.float32(1))
    d = [ux / length, uy / length, np.float32(1) / length]
    row = lambda a, k: np.broadcast_to(a[:, k, None], ux.shape)
    u = [fma32(row(M[:, k], 2), d[2], fma32(row(M[:, k], 0), d[0], row(M[:, k], 1) * d[1])) for k in range(3)]
    g = [row(g, k) for k in range(3)]
    c = [fma32(u[a], g[b], -(g[a] * u[b])) for a, b in ((1, 2), (2, 0), (0, 1))]
    norm = lambda v: fma32(v[2], v[2], fma32(v[0], v[0], v[1] * v[1])).astype(np.float64)
    alpha = opac[:, None] * np.exp(-0.5 * norm(c) / norm(u))
    kept = alpha >= 1 / 255
    clear = np.abs(alpha * 255 - 1) > 3e-6      # the hardware's division and exponential err by up to 2 and 4 roundings
    # the same in float64: pairs that the rounding of the product form decides
    u64 = [sum(M[:, k, i, None].astype(np.float64) * d[i] for i in range(3)) for k in range(3)]
    g64 = [(M[:, k].astype(np.float64) * -means).sum(-1)[:, None] for k in range(3)]
    c64 = [u64[a] * g64[b] - g64[a] * u64[b] for a, b in ((1, 2), (2, 0), (0, 1))]
    exact = opac[:, None] * np.exp(-0.5 * sum(v * v for v in c64) / sum(v * v for v in u64)) >= 1 / 255
    assert ((exact != kept) & clear).sum() >= decided

    viewmat = np.eye(4, dtype=np.float32)[None]
    K = np.array([[[f, 0, 512.0], [0, f, 512.0], [0, 0, 1]]], np.float32)
    front = (T(means), T(quats), T(scales), torch.ones((1, n, 3), device=DEV), T(opac[None]), None, None, W, H, 16, T(viewmat), None, T(K),
             pkg._capi.PINHOLE)
    lists = dict(tile_offsets=torch.arange(n, dtype=torch.int32, device=DEV).view(1, tw, tw),
                 flatten_ids=torch.arange(n, dtype=torch.int32, device=DEV))
    image, alphas, last_ids = pkg.ops.rasterize_to_pixels_from_world_3dgs_fwd(*front, **lists)
    tiles = lambda t: t.view(tw, 16, tw, 16).permute(0, 2, 1, 3).reshape(n, 256).cpu().numpy()
    got = tiles(alphas[0, ..., 0])
    assert (((got > 0) != kept) & clear).sum() == 0
    # the backward walks the same pairs: with one entry per pixel the colour's gradient is the sum of the alphas. One pair more or
    # less moves it by 3.9e-3; up to 256 float32 terms of at most 0.95 by 1e-4
    grads = pkg.ops.rasterize_to_pixels_from_world_3dgs_bwd(*front, **lists, render_alphas=alphas, last_ids=last_ids,
                                                            v_render_colors=torch.ones_like(image), v_render_alphas=torch.zeros_like(alphas))
    v_colors = grads[3][0, :, 0].cpu().numpy()
    assert np.abs(v_colors - got.astype(np.float64).sum(1)).max() < 1e-3
