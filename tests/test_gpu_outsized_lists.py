"""A large image on which a few tiles hold most of the instances: those tiles are walked with one pixel per thread by a launch of their own, the others with two.
Image and gradients against the oracle, with a distant object alone, and in front of Gaussians that give every tile a list."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NAMES = ("means", "sh0", "scaling_raw", "rotation_raw", "opacity_raw")


def T(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(DEV)


def scene(synth, W, H, behind):
    n = 3000
    rng = np.random.default_rng(W + behind)
    centre = np.array([0.011 * W, 0.006 * H, 0.0])
    near = dict(means=centre + 0.4 * rng.standard_normal((n, 3)), scaling_raw=-3.0 + 0.3 * rng.standard_normal((n, 3)))
    far = dict(means=rng.uniform(-1, 1, (behind, 3)) * [0.45 * W / 10, 0.45 * H / 10, 2.0] + [0, 0, 12.0], scaling_raw=-0.7 + 0.3 * rng.standard_normal((behind, 3)))
    P = {k: np.concatenate([near[k], far[k]]) for k in near}
    m = n + behind
    P.update(sh0=0.5 * rng.standard_normal((m, 1, 3)), shN=np.zeros((m, 0, 3)), rotation_raw=rng.standard_normal((m, 4)), opacity_raw=rng.standard_normal((m, 1)) - 1.0)
    vm = np.eye(4, dtype=np.float32)
    vm[2, 3] = 40.0
    return {k: np.ascontiguousarray(v, np.float32) for k, v in P.items()}, vm, synth.intrinsics(400.0, 400.0, W / 2.0, H / 2.0)


def check(got, want, W, H):
    # a pair at the 1/255 cut moves its pixel by 4e-3 of a colour at most
    diff = np.abs(got - want).max(-1)
    assert diff.max() < 1e-2 and (diff > 1e-4).sum() <= W * H // 500, (diff.max(), (diff > 1e-4).sum())


@pytest.mark.parametrize("W,H,behind", [(1024, 600, 0), (1024, 600, 900), (640, 480, 300), (1040, 606, 900)])   # 2,432, 2,432, 1,200 and 2,470 tiles
def test_three_linear_forms(pkg, orc, synth, W, H, behind):
    P, vm, K = scene(synth, W, H, behind)
    bg = np.array([0.2, 0.4, 0.1], np.float32)
    fwd = orc.render_fwd(P, vm, K, W, H, 0, background=bg)
    lists = np.diff(np.append(fwd["tile_offsets"].reshape(-1), fwd["flatten_ids"].size))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    share = 3 * sms if lists.size >= 16 * sms else sms // 2
    assert 0 < (lists * share > lists.sum()).sum() < 20 and (lists[lists * share <= lists.sum()] > 0).any()
    tr = pkg.trainer
    model = tr.SplatData(P["means"].shape[0], 1, DEV).load(P)
    grads, rast = model.like(), tr.Rasterizer(model, W, H, 0)
    out = rast.forward(tr.Camera(T(vm), T(K), W, H), T(bg))
    check(out.image.cpu().numpy(), fwd["render"], W, H)
    v = np.random.default_rng(1).normal(size=(H, W, 3)).astype(np.float32) * 1e-3
    bwd = orc.render_bwd(P, fwd, vm, K, W, H, 0, v, background=bg)
    rast.backward(T(v), grads, T(bg))
    for name in NAMES:
        # random output gradients cancel over the pixels of a Gaussian: a pair on the other side of the cut weighs a thousandth
        assert rel_l2(grads.tensor(name).cpu().numpy(), bwd[name]) < 2e-3, name
    # the operators have no launch order and walk all lists alike
    quats, scales, opac = orc.act_quat(P["rotation_raw"])[0], orc.act_scale(P["scaling_raw"]), orc.act_opacity(P["opacity_raw"])
    render, _, _ = pkg.ops.rasterize_to_pixels_from_world_3dgs_fwd(
        T(P["means"]), T(quats), T(scales), T(fwd["colors"][None]), T(opac[None]), T(bg[None]), None, W, H, 16, T(vm[None]), None, T(K[None]), 0,
        tile_offsets=torch.from_numpy(fwd["tile_offsets"][None]).to(DEV), flatten_ids=torch.from_numpy(fwd["flatten_ids"]).to(DEV))
    check(render.cpu().numpy()[0], fwd["render"], W, H)


@pytest.mark.parametrize("W,H,behind", [(1040, 606, 0), (1040, 606, 900), (640, 480, 300)])   # 2,470 tiles (two pixels in both directions) and 1,200 (backward)
def test_ewa(pkg, orc, synth, W, H, behind):
    P, vm, K = scene(synth, W, H, behind)
    bg = np.array([0.2, 0.4, 0.1], np.float32)
    campos = orc.campos(vm)
    fwd = orc.ewa_forward(P, vm, campos, W, H, K[0, 0], K[1, 1], K[0, 2], K[1, 2], 1, background=bg)
    tr = pkg.trainer
    model = tr.SplatData(P["means"].shape[0], 1, DEV).load(P)
    grads, rast = model.like(), tr.FastRasterizer(model, W, H, 0)
    out = rast.forward(tr.Camera(T(vm), T(K), W, H), T(bg), cam_position=T(np.asarray(campos, np.float32)))
    check(out.image.cpu().numpy().transpose(1, 2, 0), fwd["image"].transpose(1, 2, 0), W, H)
    v = np.random.default_rng(1).normal(size=(3, H, W)).astype(np.float32) * 1e-3
    bwd = orc.ewa_backward(P, fwd, v)
    rast.backward(T(v), grads, T(bg))
    for name in NAMES:
        assert rel_l2(grads.tensor(name).cpu().numpy(), bwd[name]) < 2e-3, name


# the two launches side by side inside a CUDA graph, replayed on other inputs than it was captured with
@pytest.mark.parametrize("ewa", [False, True])
def test_captured(pkg, synth, ewa):
    W, H = 1040, 606
    tr = pkg.trainer
    (P, vm, K), (Q, _, _) = scene(synth, W, H, 900), scene(synth, W, H, 901)
    Q = {k: np.concatenate([v[:3000], v[3001:]]) for k, v in Q.items()}
    model = tr.SplatData(3900, 1, DEV).load(P)
    rast, grads = (tr.FastRasterizer if ewa else tr.Rasterizer)(model, W, H, 0), model.like()
    cam, bg = tr.Camera(T(vm), T(K), W, H), torch.zeros(3, device=DEV)
    v = torch.full((3, H, W) if ewa else (H, W, 3), 1e-3, device=DEV)

    def step():
        out = rast.forward(cam, bg)
        rast.backward(v, grads, bg)
        return out.image

    def results():
        return [x.clone() for x in (image, *(grads.tensor(n) for n in NAMES))]

    for _ in range(2):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        image = step()
    model.load(Q)
    graph.replay()
    torch.cuda.synchronize()
    replayed = results()
    image = step()
    for a, b in zip(replayed, results()):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 1e-5    # gradients: sums in another order
    assert torch.equal(replayed[0], image)
    del graph
