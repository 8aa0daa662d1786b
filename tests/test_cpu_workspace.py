"""Workspace sizes. Programs size a workspace once for the capacity of their model and call with every smaller number of Gaussians, so
no size may fall as a count grows, also not where the list sorts change their method (2,097,152 Gaussians, 6,291,456 instances)."""
import ctypes as C

import pytest

COUNTS = sorted({1, 255, 2049, 70_001, 1_000_000, *(m + d for m in (2_097_152, 6_291_456) for d in (-20_000, -2048, -1, 0, 1, 2, 2049, 40_000))})


def _render(pkg, n, capacity, ewa):
    capi = pkg._capi
    cfg = capi.EwaConfig() if ewa else capi.RenderConfig()
    cfg.N, cfg.sh_coeffs, cfg.image_width, cfg.image_height = n, 16, 1296, 840
    if ewa:
        cfg.active_sh_bases, cfg.focal_x, cfg.focal_y, cfg.near_plane, cfg.far_plane = 16, 1.0, 1.0, 0.01, 1e10
        cfg.instance_capacity = capacity
        return capi.lib().lfs_ewa_workspace_bytes(C.byref(cfg))
    cfg.sh_degree, cfg.tile_size, cfg.eps2d, cfg.far_plane, cfg.isect_capacity = 3, 16, 0.3, 1e10, capacity
    cfg.shutter, cfg.scaling_modifier = 0, 1.0
    return capi.lib().lfs_render_workspace_bytes(C.byref(cfg))


@pytest.mark.parametrize("name", ["render", "ewa", "operator"])
@pytest.mark.parametrize("grows", ["gaussians", "instances"])
def test_workspace_sizes_never_fall(pkg, name, grows):
    def size(n, capacity):
        if name == "operator":
            return pkg._capi.lib().lfs_intersect_tile_workspace_bytes(1, n, capacity)
        return _render(pkg, n, capacity, name == "ewa")

    sizes = [size(n, 100_000) if grows == "gaussians" else size(1000, n) for n in COUNTS]
    assert sizes[0] > 0 and all(a <= b for a, b in zip(sizes, sizes[1:])), list(zip(COUNTS, sizes))
