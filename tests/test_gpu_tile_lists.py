"""Tile lists against a stable host sort of the same instances: lists on both sides of every size at which the sorting groups change, depths that
defeat the buckets (equal, few, one far away, negative), rectangles larger than a warp, several cameras, more tiles than one round holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
F = np.float32


def _instances(m, r, d, ts, tw, th):
    """(64-bit key, flattened index) of every instance in emission order."""
    keys, ids = [], []
    C, N = d.shape
    for c in range(C):
        lo = [np.minimum(np.maximum(np.floor(m[c, :, a] / F(ts) - r[c, :, a].astype(F) / F(ts)), 0), n).astype(np.int64) for a, n in ((0, tw), (1, th))]
        hi = [np.minimum(np.maximum(np.ceil(m[c, :, a] / F(ts) + r[c, :, a].astype(F) / F(ts)), 0), n).astype(np.int64) for a, n in ((0, tw), (1, th))]
        w = hi[0] - lo[0]
        n = np.where((r[c] > 0).all(-1), w * (hi[1] - lo[1]), 0)
        g = np.repeat(np.arange(N), n)
        local = np.arange(n.sum()) - (np.cumsum(n) - n)[g]
        tile = (lo[1][g] + local // np.maximum(w[g], 1)) * tw + lo[0][g] + local % np.maximum(w[g], 1)
        depth = d[c].view(np.uint32).astype(np.int64)[g]
        keys.append((((c << int(tw * th).bit_length()) | tile) << 32) | depth)
        ids.append(g + c * N)
    return np.concatenate(keys), np.concatenate(ids)


def _check(pkg, m, r, d, tw, th, ts=16):
    m, r, d = m.astype(F), r.astype(np.int32), d.astype(F)
    keys, ids = _instances(m, r, d, ts, tw, th)
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (m, r, d)]
    for sort in (True, False):
        _, k, i = pkg.ops.intersect_tile(*t, None, None, d.shape[0], ts, tw, th, sort)
        o = np.argsort(keys, kind="stable") if sort else slice(None)
        assert np.array_equal(k.cpu().numpy(), keys[o]) and np.array_equal(i.cpu().numpy(), ids[o])


DEPTHS = {
    "spread": lambda rng, n: rng.random(n) * 5 + 0.5,
    "equal": lambda rng, n: np.full(n, 3.25),
    "few": lambda rng, n: rng.integers(1, 5, n).astype(float),
    "far": lambda rng, n: np.concatenate([[9000.0], rng.random(n - 1) * 1e-3 + 2]),
    "negative": lambda rng, n: rng.standard_normal(n),
}


@pytest.mark.parametrize("depths", DEPTHS)
@pytest.mark.parametrize("n", [1, 31, 33, 127, 128, 129, 255, 256, 512, 513, 1023, 1024, 2047, 2048, 2049, 4096, 4097, 8191, 8192, 8193, 9000, 70_001])
def test_one_list(pkg, n, depths):
    d = DEPTHS[depths](np.random.default_rng(n), n)
    _check(pkg, np.full((1, n, 2), 8.0), np.ones((1, n, 2)), d[None], 1, 1)


@pytest.mark.parametrize("C,N,tw,th,ts,radius", [
    (1, 20_000, 40, 27, 16, 30),      # lists of all the sizes
    (2, 5000, 13, 9, 16, 60),
    (5, 2000, 1, 1, 16, 4),
    (1, 30, 700, 600, 16, 6000),      # rectangles of thousands of tiles; 420,000 tiles: four rounds
    (3, 300, 500, 400, 4, 300),       # rounds that end inside a camera
    (1, 100_000, 3, 2, 16, 12),
])
def test_many_lists(pkg, C, N, tw, th, ts, radius):
    rng = np.random.default_rng(N)
    m = rng.random((C, N, 2)) * [tw * ts, th * ts]
    _check(pkg, m, rng.integers(0, radius, (C, N, 2)), np.exp(rng.standard_normal((C, N))), tw, th, ts)


# Lists of 65,536 entries and more among more than 262,144 Gaussians are cut into bins by drawn limits first. Twelve million: bins beyond the sorting room.
@pytest.mark.parametrize("n,depths,tiles", [(262_144, "spread", 1), (262_145, "spread", 1), (262_145, "equal", 1), (262_145, "few", 1), (262_145, "far", 1),
                                            (262_145, "negative", 1), (300_007, "far", 3), (500_000, "spread", 7), (1_200_000, "far", 9), (1_000_003, "far", 1), (12_000_000, "spread", 1)])
def test_far_lists(pkg, n, depths, tiles):
    rng = np.random.default_rng(n)
    d = torch.from_numpy(DEPTHS[depths](rng, n).astype(F)).cuda()
    tile = torch.arange(n, device="cuda") % (n if tiles == 1 else 9) % tiles      # of seven tiles two hold twice as much as the others
    m = torch.stack([16.0 * tile + 8.0, torch.full((n,), 8.0, device="cuda")], -1)[None].float().contiguous()
    r = torch.ones((1, n, 2), dtype=torch.int32, device="cuda")
    _, k, i = pkg.ops.intersect_tile(m, r, d[None].contiguous(), None, None, 1, 16, tiles, 1, True)
    key = (tile << 32) | (d.view(torch.int32).long() & 0xFFFFFFFF)
    order = torch.sort(key, stable=True).indices
    assert torch.equal(k, key[order]) and torch.equal(i.long(), order)


# A Gaussian behind the camera makes far lists possible; it must not make a difference. Some 330,000 entries in a tile among the 262,144 or 262,145.
@pytest.mark.parametrize("ewa", [False, True])
def test_far_lists_of_a_render(pkg, synth, ewa):
    n, W, H = 262_144, 96, 64
    P = synth.make_gaussians(n + 1, 5, "cube", 0)
    P["means"][n] = [0.0, -400.0, 0.0]
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a, F)).cuda()
    tr = pkg.trainer
    cam = tr.Camera(T(synth.look_at_origin([0.3, -40.0, 0.4])), T(synth.intrinsics(200.0, 200.0, 40.0, 24.0)), W, H)
    images = []
    for count in (n, n + 1):
        model = tr.SplatData(count, 1, "cuda:0").load({k: v[:count] for k, v in P.items()})
        rast = (tr.FastRasterizer if ewa else tr.Rasterizer)(model, W, H, 0)
        images.append(rast.forward(cam, None).image.clone())
        if not ewa:
            assert (torch.diff(rast.state()["tile_offsets"]) >= 65_536).any()
    assert images[0].abs().max() > 0.1 and torch.equal(*images)


# The fused path counts the instances in the projection, or, where few Gaussians face many tiles (eight tiles a Gaussian or more while several warps share
# 32 of them, up to 75,776 on 148 SMs), in a launch of its own: 192 and 9,600 tiles, a Gaussian on either side of each limit.
@pytest.mark.parametrize("n,W,H", [(1535, 256, 192), (1536, 256, 192), (1537, 256, 192), (75_776, 1920, 1280), (75_777, 1920, 1280)])
def test_lists_of_a_render(pkg, synth, n, W, H):
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a, F)).cuda()
    tr = pkg.trainer
    model = tr.SplatData(n, 1, "cuda:0").load(synth.make_gaussians(n, 2, "cube", 0))
    rast = tr.Rasterizer(model, W, H, 0, isect_capacity=1 << 22)
    rast.forward(tr.Camera(T(synth.look_at_origin([0.3, -4.0, 0.4])), T(synth.intrinsics(1.1 * W, 1.1 * W, W / 2, H / 2)), W, H), None)
    st = {k: v.cpu().numpy() for k, v in rast.state().items() if torch.is_tensor(v)}
    tw, th = W // 16, H // 16
    keys, ids = _instances(st["means2d"][None], st["radii"][None], st["depths"][None], 16, tw, th)
    order = np.argsort(keys, kind="stable")
    assert ids.size > 2 * n and np.array_equal(st["flatten_ids"], ids[order])
    assert np.array_equal(st["tile_offsets"], np.searchsorted(keys[order] >> 32, np.arange(tw * th + 1)))
