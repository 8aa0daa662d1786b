"""The fisheye projection takes the angles of a Gaussian's sigma points from the first one's (angle_near of csrc/gsmath.cuh): points that nearly coincide,
points on both sides of the limit of its series, points on the optical axis and far from it, against the oracle's arc tangents. The two angles agree to some
2^-51, so a float rounds differently about once in 10^8 points: none of the some 4 10^5 here."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.01, 0.05, 0.3, 2.0])
@pytest.mark.parametrize("place", ["ahead", "axis", "edge", "close"])
def test_sigma_points(pkg, orc, scale, place):
    n, W, H = 4001, 640, 480
    rng = np.random.default_rng(int(scale * 100) + len(place))
    direction = rng.standard_normal((n, 3)) * {"ahead": 1.0, "axis": 1e-4, "edge": 1.0, "close": 1.0}[place]
    if place == "edge":
        direction[:, 2] = np.abs(direction[:, 2]) * 0.02
    else:
        direction[:, 2] = np.abs(direction[:, 2]) + (1.0 if place == "axis" else 0.1)
    means = direction / np.linalg.norm(direction, axis=1, keepdims=True) * (0.2 if place == "close" else 4.0) * (1 + rng.random((n, 1)))
    quats = rng.standard_normal((n, 4))
    quats /= np.linalg.norm(quats, axis=1, keepdims=True)
    arrays = [np.ascontiguousarray(x, np.float32) for x in (means, quats, scale * np.exp(0.5 * rng.standard_normal((n, 3))), 0.2 + 0.7 * rng.random(n))]
    vm, K = np.eye(4, dtype=np.float32)[None], np.array([[[W / np.pi, 0, W / 2], [0, W / np.pi, H / 2], [0, 0, 1]]], np.float32)
    ref = orc.projection_ut_3dgs_fused(*arrays, vm, K, W, H, camera_model=2)
    t = [torch.from_numpy(a).cuda() for a in (*arrays, vm, K)]
    radii, means2d, depths, conics, _ = pkg.ops.projection_ut_3dgs_fused(*t[:4], t[4], None, t[5], W, H, 0.3, 0.01, 1e4, 0.0, False, 2)
    assert np.array_equal(radii.cpu().numpy(), ref[0])
    vis = (ref[0][0] > 0).all(-1)
    assert vis.sum() > 100
    for got, want in ((means2d, ref[1]), (depths, ref[2]), (conics, ref[3])):
        assert np.array_equal(got.cpu().numpy()[0][vis].view(np.uint32), want[0][vis].view(np.uint32))


# distances of 2e17 to 1e20: the products of two points lie on both sides of the largest float, whose reciprocal starts the division
@pytest.mark.parametrize("scale", [0.01, 0.05, 0.3])
def test_remote_sigma_points(pkg, orc, scale):
    n, W, H, far = 4001, 640, 480, 1e30
    rng = np.random.default_rng(int(scale * 100))
    direction = rng.standard_normal((n, 3))
    direction[:, 2] = np.abs(direction[:, 2]) + 0.1
    distance = 10.0 ** rng.uniform(17.3, 20.0, (n, 1))
    quats = rng.standard_normal((n, 4))
    means, scales = direction / np.linalg.norm(direction, axis=1, keepdims=True) * distance, 0.25 * scale * distance * np.exp(0.5 * rng.standard_normal((n, 3)))
    arrays = [np.ascontiguousarray(x, np.float32) for x in (means, quats / np.linalg.norm(quats, axis=1, keepdims=True), scales, 0.2 + 0.7 * rng.random(n))]
    vm, K = np.eye(4, dtype=np.float32)[None], np.array([[[W / np.pi, 0, W / 2], [0, W / np.pi, H / 2], [0, 0, 1]]], np.float32)
    ref = orc.projection_ut_3dgs_fused(*arrays, vm, K, W, H, far=far, camera_model=2)
    t = [torch.from_numpy(a).cuda() for a in (*arrays, vm, K)]
    radii, means2d, _, conics, _ = pkg.ops.projection_ut_3dgs_fused(*t[:4], t[4], None, t[5], W, H, 0.3, 0.01, far, 0.0, False, 2)
    assert np.array_equal(radii.cpu().numpy(), ref[0])
    vis = (ref[0][0] > 0).all(-1)
    assert vis.sum() > 100
    for got, want in ((means2d, ref[1]), (conics, ref[3])):
        assert np.array_equal(got.cpu().numpy()[0][vis].view(np.uint32), want[0][vis].view(np.uint32))
