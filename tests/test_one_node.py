"""Scenes whose tree is one node (their rays take a kernel of their own): every
primitive kind, transformed and moving ones, at ray counts around a warp, in
both modes, against the CPU oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def small_scene(ptgb, kind, w, h):
    s = ptgb.Scene()
    a, b = s.lambertian((0.7, 0.6, 0.5)), s.metal((0.8, 0.8, 0.9), 0.1)
    glow = s.diffuse_light((4.0, 4.0, 3.0))
    s.miss_gradient((1.0, 1.0, 1.0), (0.5, 0.7, 1.0))
    if kind == "one":
        s.sphere((0.0, 0.0, 0.0), 0.7, a)
    else:
        xf = ptgb.compose([ptgb.mat_translate((0.6, 0.1, -0.4)), ptgb.mat_rotate(25.0, 1)])
        s.box((-0.3, -0.3, -0.3), (0.3, 0.4, 0.3), a, xf)
        s.rect(-2, 2, -2, 2, -0.6, False, ptgb.PT_Y_AXIS, a)
        s.sphere((-0.6, 0.0, 0.2), 0.4, b)
        if kind == "motion":
            s.moving_sphere((0.0, 0.6, 0.0), (0.3, 0.8, 0.0), 0.25, 0.0, 1.0, a)
        tri = np.array([[-1, -0.6, -1], [1, -0.6, -1], [0, 1.2, -1.2]], np.float32)
        s.mesh(tri, np.arange(3, dtype=np.uint32), s.oren_nayar((0.6, 0.7, 0.6), 0.4))
        s.rect(-0.5, 0.5, -0.5, 0.5, 1.9, True, ptgb.PT_Y_AXIS, glow)
        s.light_rect(-0.5, 0.5, -0.5, 0.5, 1.9, ptgb.PT_Y_AXIS, (4.0, 4.0, 3.0))
    s.set_camera((0.3, 0.5, 3.0), (0, 0, 0), (0, 1, 0), 50.0, w / h, 0.05, 3.0, 0.0, 1.0)
    return s


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kind", ["one", "mixed", "motion"])
@pytest.mark.parametrize("w,h,slots", [(1, 1, 0), (31, 1, 0), (33, 2, 0), (131, 127, 0), (131, 127, 999)])
def test_one_node_scenes(ptgb_mod, oracle_mod, kind, mode, w, h, slots):
    s = small_scene(ptgb_mod, kind, w, h)
    g, o = ptgb_mod.GpuRenderer(s, path_slots=slots), oracle_mod.Oracle(s)
    assert g.stats()["bvh_nodes"] == 1
    for a, b in zip(g.first_hits(w, h, 3), o.first_hits(w, h, 3)):
        assert np.array_equal(a, b)
    gpu = g.render_paths(ptgb_mod.GpuRenderer.params(w, h, 1, frame0=2, mode=mode)).reshape(-1, 3)
    assert np.array_equal(gpu, o.render_paths(w, h, 2, np.arange(w * h), mode=mode))
    g.close()
