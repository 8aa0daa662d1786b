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


# ---- boxes and patches: one Gaussian per tile list, every pair against float64 -----------------------------------------
def _quat(R):
    """float32 quaternions (w, x, y, z) of rotation matrices [n, 3, 3]"""
    q = np.sqrt(np.maximum(0, 1 + np.stack([R[:, 0, 0] + R[:, 1, 1] + R[:, 2, 2], R[:, 0, 0] - R[:, 1, 1] - R[:, 2, 2],
                                            R[:, 1, 1] - R[:, 0, 0] - R[:, 2, 2], R[:, 2, 2] - R[:, 0, 0] - R[:, 1, 1]], -1))) / 2
    q[:, 1] = np.copysign(q[:, 1], R[:, 2, 1] - R[:, 1, 2])
    q[:, 2] = np.copysign(q[:, 2], R[:, 0, 2] - R[:, 2, 0])
    q[:, 3] = np.copysign(q[:, 3], R[:, 1, 0] - R[:, 0, 1])
    return q.astype(np.float32)


def _rotmat(q):
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                     [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                     [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]]).transpose(2, 0, 1)


def _alpha64(means, quats, scales, opac, owner, d):
    """[H, W] alpha of each pixel's own Gaussian (owner, -1 = none) along the line of its ray d [H, W, 3]"""
    M = _rotmat(quats.astype(np.float64)).transpose(0, 2, 1) / scales.astype(np.float64)[:, :, None]
    g = (M @ -means.astype(np.float64)[:, :, None])[:, :, 0]
    at = np.maximum(owner, 0)
    u = np.einsum("hwij,hwj->hwi", M[at], d)
    c = np.cross(u, g[at])
    return np.where(owner >= 0, opac[at] * np.exp(-0.5 * (c * c).sum(-1) / (u * u).sum(-1)), 0.0)


def _check_single_lists(pkg, means, quats, scales, opac, tile_owner, W, H, f):
    """Equidistant fisheye at the origin. Every pair with alpha clearly above 1/255 is blended, none clearly below, and the backward
    walks the same pairs."""
    n, th, tw = len(means), H // 16, W // 16
    j, i = np.meshgrid(np.arange(W) + 0.5, np.arange(H) + 0.5)
    ux, uy = (j - W / 2) / f, (i - H / 2) / f
    theta = np.hypot(ux, uy)
    d = np.stack([np.sin(theta) / theta * ux, np.sin(theta) / theta * uy, np.cos(theta)], -1)
    owner = np.repeat(np.repeat(tile_owner, 16, 0), 16, 1)
    alpha = _alpha64(means, quats, scales, opac, owner, d)
    valid = theta < np.hypot(W / 2, H / 2) / f * (1 - 1e-6)
    K = np.array([[[f, 0, W / 2], [0, f, H / 2], [0, 0, 1]]], np.float32)
    front = (T(means), T(quats), T(scales), torch.ones((1, n, 3), device=DEV), T(opac[None]), None, None, W, H, 16,
             T(np.eye(4, dtype=np.float32)[None]), None, T(K), pkg._capi.FISHEYE)
    has = tile_owner.reshape(-1) >= 0
    lists = dict(tile_offsets=T((np.cumsum(has) - has).astype(np.int32).reshape(1, th, tw)),
                 flatten_ids=T(tile_owner.reshape(-1)[has].astype(np.int32)))
    radial = torch.zeros((1, 4), device=DEV)
    image, alphas, last_ids = pkg.ops.rasterize_to_pixels_from_world_3dgs_fwd(*front, radial_coeffs=radial, **lists)
    got = alphas[0, ..., 0].cpu().numpy().astype(np.float64)
    # the kernels' float32 response errs by a few 2^-24 (distance / smallest scale): 2 % where that ratio is 1e4 or less
    assert (1 / scales.min(1) * np.linalg.norm(means, axis=1)).max() < 1e4
    lost, extra = valid & (alpha > 1.02 / 255) & (got == 0), (alpha < 0.98 / 255) & (got > 0)
    assert lost.sum() == 0 and extra.sum() == 0, (lost.sum(), alpha[lost].max() if lost.any() else 0, extra.sum())
    grads = pkg.ops.rasterize_to_pixels_from_world_3dgs_bwd(*front, radial_coeffs=radial, **lists, render_alphas=alphas, last_ids=last_ids,
                                                            v_render_colors=torch.ones_like(image), v_render_alphas=torch.zeros_like(alphas))
    # one entry per pixel: the colour's gradient is the sum of the blended alphas. A pair more or less moves it by 3.9e-3 and more, the
    # float32 sum of up to 3e4 alphas by their rounding
    total = np.array([got[owner == g].sum() for g in range(n)])
    assert np.abs(grads[3][0, :, 0].cpu().numpy() - total).max() < 2e-3 + 2e-6 * total.max()


# needles that point at the camera and reach close to it: sixty to a thousand times longer than wide, twice to ten times wider than thick
@pytest.mark.parametrize("seed", range(4))
def test_fisheye_keeps_the_pairs_of_needles_along_the_ray(pkg, seed):
    rng = np.random.default_rng(seed)
    W = H = 2048
    block = 8                                   # tiles of a needle's own square
    by, bx = np.divmod(np.arange(256), 16)
    f = 1400.0                                  # 84 degrees across the image
    px = np.stack([bx * 128 + 64 + rng.uniform(-8, 8, 256), by * 128 + 64 + rng.uniform(-8, 8, 256)], -1)
    u = (px - 1024) / f
    theta = np.linalg.norm(u, axis=1)
    e = np.stack([np.sin(theta) / theta * u[:, 0], np.sin(theta) / theta * u[:, 1], np.cos(theta)], -1)
    n = len(e)
    dist = np.exp(rng.uniform(-1, 1, n))
    opac = rng.uniform(0.3, 0.95, n).astype(np.float32)
    length = dist * rng.uniform(0.5, 0.98, n) / np.sqrt(2 * np.log(255 * opac))
    width = length / 10 ** rng.uniform(1.8, 2.3, n)
    scales = np.stack([length, width, np.maximum(width * rng.uniform(0.1, 0.5, n), dist / 9000)], -1).astype(np.float32)
    a = e + 10 ** rng.uniform(-6, -4, (n, 1)) * rng.normal(size=(n, 3))
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b = np.cross(a, rng.normal(size=(n, 3)))
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    quats = _quat(np.stack([a, b, np.cross(a, b)], -1))
    owner = np.arange(256).reshape(16, 16).repeat(block, 0).repeat(block, 1)
    _check_single_lists(pkg, (e * dist[:, None]).astype(np.float32), quats, scales, opac, owner, W, H, f)


# A lens that sees past the plane of the camera: a Gaussian also answers the rays that leave it behind them
@pytest.mark.parametrize("fov", [150, 180, 200, 220, 270])
def test_fisheye_keeps_the_pairs_behind_the_ray(pkg, fov):
    rng = np.random.default_rng(fov)
    W = H = 256
    n = 24
    f = W / np.radians(fov)
    e = rng.normal(size=(n, 3))
    e /= np.linalg.norm(e, axis=1, keepdims=True)
    dist = np.exp(rng.uniform(-1, 1, n))
    scales = (dist[:, None] * np.exp(-2.2 + 0.6 * rng.normal(size=(n, 3)))).astype(np.float32)
    q = rng.normal(size=(n, 4))
    quats = (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)
    opac = rng.uniform(0.1, 0.95, n).astype(np.float32)
    means = (e * dist[:, None]).astype(np.float32)
    for g in range(n):
        one = slice(g, g + 1)
        _check_single_lists(pkg, means[one], quats[one], scales[one], opac[one], np.zeros((H // 16, W // 16), int), W, H, f)


@pytest.mark.parametrize("n,fov,grow,fade", [(20000, 180, 1.2, 0.0), (20000, 200, 1.0, 0.0), (1000, 220, 2.2, 2.0)])
def test_fisheye_inside_a_scene(pkg, orc, synth, n, fov, grow, fade):
    tr, capi = pkg.trainer, pkg._capi
    W = H = 256
    deg = 1
    P = synth.make_gaussians(n, 5, "cube", deg)
    P["scaling_raw"] = (P["scaling_raw"] + np.float32(grow)).astype(np.float32)
    P["opacity_raw"] = (P["opacity_raw"] - np.float32(fade)).astype(np.float32)
    vm = synth.look_at_origin([0.1, -0.2, 0.1])
    f = min(W, H) / np.radians(fov)
    K = synth.intrinsics(f, f, W / 2.0, H / 2.0)
    radial = np.zeros(4, np.float32)
    kw = dict(camera_model=orc.FISHEYE, radial=radial)
    fwd = orc.render_fwd(P, vm, K, W, H, deg, **kw)
    model = tr.SplatData(n, (deg + 1) ** 2, DEV).load(P)
    grads = model.like()
    rast = tr.Rasterizer(model, W, H, deg, camera_model=capi.FISHEYE)
    out = rast.forward(tr.Camera(T(vm), T(K), W, H, capi.FISHEYE, radial=T(radial)), None)
    diff = np.abs(out.image.cpu().numpy() - fwd["render"]).max(-1)
    # The oracle rounds the product form without fused operations: a pair within that of the cut falls on either side, 4e-3 of a colour
    # of up to 1.5 in a pixel here and there. Lost cones show as larger differences or in many pixels
    assert diff.max() < 8e-3 and (diff > 1e-4).sum() <= 20, (diff.max(), (diff > 1e-4).sum())
    rng = np.random.default_rng(1)
    v_r, v_a = (rng.normal(size=(H, W, k)).astype(np.float32) * 1e-3 for k in (3, 1))
    bwd = orc.render_bwd(P, fwd, vm, K, W, H, deg, v_r, v_a, **kw)
    rast.backward(T(v_r), grads, None, T(v_a))
    for name in ("means", "sh0", "shN", "scaling_raw", "rotation_raw", "opacity_raw"):
        assert rel_l2(grads.tensor(name).cpu().numpy(), bwd[name]) < 2e-3, name   # as at the backward's other parity tests


# Lenses whose inversion runs away to infinity in pixels that share a warp's patch with valid ones (some two dozen of them each)
@pytest.mark.parametrize("rolling", [False, True])
@pytest.mark.parametrize("k,f", [((-0.0813082829, -0.525065839, 0.20530051), 111.764832), ((-0.119644128, -0.4756459, 0.237992167), 85.6079636),
                                 ((-0.101954706, -0.259541839, 0.101956189), 70.9386826)])
def test_pixels_without_a_ray_leave_the_gradients_finite(pkg, synth, k, f, rolling):
    tr, capi = pkg.trainer, pkg._capi
    n, W, H, deg = 3000, 208, 144, 1
    P = synth.make_gaussians(n, 7, "cube", deg)
    vm = synth.look_at_origin([0.3, -2.0, 0.4])
    K = synth.intrinsics(f, f, W / 2.0, H / 2.0)
    radial = np.zeros(6, np.float32)
    radial[:3] = k
    model = tr.SplatData(n, (deg + 1) ** 2, DEV).load(P)
    grads = model.like()
    rast = tr.Rasterizer(model, W, H, deg)
    end = dict(viewmat_end=T(synth.look_at_origin([0.31, -2.0, 0.4])), shutter=1) if rolling else {}
    out = rast.forward(tr.Camera(T(vm), T(K), W, H, radial=T(radial), **end), None)
    assert torch.isfinite(out.image).all()
    rast.backward(torch.full((H, W, 3), 1e-3, device=DEV), grads, None)
    for name in ("means", "sh0", "shN", "scaling_raw", "rotation_raw", "opacity_raw"):
        g = grads.tensor(name)
        assert torch.isfinite(g).all() and g.abs().max() > 0, name


# A Gaussian centred on the camera answers every ray with its opacity, in front of the camera or behind it
@pytest.mark.parametrize("fisheye", [False, True])
def test_camera_on_the_centre(pkg, fisheye):
    W = H = 512
    tiles = (W // 16) * (H // 16)
    one = lambda *v: torch.tensor([v], dtype=torch.float32, device=DEV)
    eye = torch.eye(4, device=DEV)[None]
    lists = dict(tile_offsets=torch.arange(tiles, dtype=torch.int32, device=DEV).view(1, H // 16, W // 16),
                 flatten_ids=torch.zeros(tiles, dtype=torch.int32, device=DEV))
    if fisheye:
        lists["radial_coeffs"] = torch.zeros((1, 4), device=DEV)
    for shift in range(2):
        f = W / 3.5 if fisheye else W / 3.0
        K = torch.tensor([[[f, 0, W / 2 + 0.37 * shift], [0, f, H / 2 - 0.21 * shift], [0, 0, 1]]], device=DEV)
        front = (one(0, 0, 0), one(0.8, 0.2, -0.4, 0.4), one(0.3, 0.2, 0.1), torch.ones((1, 1, 3), device=DEV), one(0.5), None, None, W, H, 16,
                 eye, None, K, pkg._capi.FISHEYE if fisheye else pkg._capi.PINHOLE)
        image, alphas, last_ids = pkg.ops.rasterize_to_pixels_from_world_3dgs_fwd(*front, **lists)
        inside = alphas > 0 if fisheye else torch.ones_like(alphas, dtype=torch.bool)   # a fisheye's corners have no ray
        assert inside.float().mean() > 0.7 and (alphas[inside] == 0.5).all()
        grads = pkg.ops.rasterize_to_pixels_from_world_3dgs_bwd(*front, **lists, render_alphas=alphas, last_ids=last_ids,
                                                                v_render_colors=torch.ones_like(image), v_render_alphas=torch.zeros_like(alphas))
        assert all(torch.isfinite(g).all() for g in grads)
        assert (grads[0] == 0).all() and (grads[2] == 0).all()


# Large Gaussians close to a strongly distorted pinhole, image and gradients: the backward's patches have another shape than the forward's.
# Every pixel's ray converges: where the inversion hardly does, fused operations decide whether a pixel has one.
@pytest.mark.parametrize("k,f,dist,grow", [([-0.3, 0.12, -0.02, 0.01, 0.0, 0.0], 200.0, 1.5, 0.8), ([0.25, 0.05, 0.0, 0.0, 0.02, 0.0], 120.0, 2.2, 0.3),
                                           ([-0.2, 0.05, 0.0, 0.0, 0.0, 0.0], 300.0, 1.2, 1.0)])
def test_distorted_pinhole_close_to_a_scene(pkg, orc, synth, k, f, dist, grow):
    tr = pkg.trainer
    n, W, H, deg = 6000, 308, 236, 1
    P = synth.make_gaussians(n, 3, "cube", deg)
    P["scaling_raw"] = (P["scaling_raw"] + np.float32(grow)).astype(np.float32)
    vm = synth.look_at_origin([0.3, -dist, 0.4])
    K = synth.intrinsics(f, f * 0.97, W / 2 + 5.0, H / 2 - 3.0)
    radial, tangential = np.array(k, np.float32), np.array([1e-3, -5e-4], np.float32)
    packed = orc.pack_distortion(radial=radial, tangential=tangential)
    fwd = orc.render_fwd(P, vm, K, W, H, deg, radial=packed)
    model = tr.SplatData(n, (deg + 1) ** 2, DEV).load(P)
    grads = model.like()
    rast = tr.Rasterizer(model, W, H, deg)
    out = rast.forward(tr.Camera(T(vm), T(K), W, H, radial=T(radial), tangential=T(tangential)), None)
    diff = np.abs(out.image.cpu().numpy() - fwd["render"]).max(-1)
    assert diff.max() < 8e-3 and (diff > 1e-4).sum() <= 20, (diff.max(), (diff > 1e-4).sum())   # pairs at the cut, as above
    rng = np.random.default_rng(1)
    v_r, v_a = (rng.normal(size=(H, W, c)).astype(np.float32) * 1e-3 for c in (3, 1))
    bwd = orc.render_bwd(P, fwd, vm, K, W, H, deg, v_r, v_a, radial=packed)
    rast.backward(T(v_r), grads, None, T(v_a))
    for name in ("means", "sh0", "shN", "scaling_raw", "rotation_raw", "opacity_raw"):
        assert rel_l2(grads.tensor(name).cpu().numpy(), bwd[name]) < 2e-3, name
