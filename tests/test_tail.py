"""The tail kernel (the last paths of a chunk, each traced to its end by one
thread) against the CPU oracle, at the sizes where a chunk goes to it whole,
just misses it, or reaches it from the wavefront."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL_TOL = 1e-4  # the parity contract of the path tracer


def rel_err(a, b):
    return np.abs(a - b) / np.maximum(np.maximum(np.abs(a), np.abs(b)), 1e-3)


# 16384 paths and fewer are one tail launch; 129 x 128 is the first size past it
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("w,h,spp,slots", [(1, 1, 1, 0), (33, 1, 1, 0), (128, 128, 1, 0),
                                           (129, 128, 1, 0), (64, 48, 11, 0), (64, 48, 6, 1000)])
def test_tail_sizes(ptgb_mod, oracle_mod, mode, w, h, spp, slots):
    s = ptgb_mod.material_zoo(w, h)
    g, o = ptgb_mod.GpuRenderer(s, path_slots=slots), oracle_mod.Oracle(s)
    acc = g.render(ptgb_mod.GpuRenderer.params(w, h, spp, mode=mode))
    ref, st = o.render(w, h, spp, mode=mode)
    assert np.array_equal(acc[..., 3], ref[..., 3])
    assert rel_err(acc[..., :3], ref[..., :3]).max() <= REL_TOL
    gs = g.stats()
    assert gs["ext_rays"] == st["ext_rays"] and gs["shadow_rays"] == st["shadow_rays"]
    # with stage timing the same kernels run under the host loop
    t = ptgb_mod.GpuRenderer(s, path_slots=slots, timing=True, counters=True)
    assert np.array_equal(t.render(ptgb_mod.GpuRenderer.params(w, h, spp, mode=mode)), acc)
    ts = t.stats()
    assert ts["ext_rays"] == gs["ext_rays"] and ts["node_fetches"] > 0
    g.close()
    t.close()


# with image or noise textures 4096 paths and fewer are one tail launch
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("w", [64, 65])
def test_tail_sizes_textured(ptgb_mod, oracle_mod, mode, w):
    s = ptgb_mod.texture_zoo(w, 64)
    g, o = ptgb_mod.GpuRenderer(s), oracle_mod.Oracle(s)
    acc = g.render(ptgb_mod.GpuRenderer.params(w, 64, 1, mode=mode))
    ref, st = o.render(w, 64, 1, mode=mode)
    assert np.array_equal(acc[..., 3], ref[..., 3])
    assert rel_err(acc[..., :3], ref[..., :3]).max() <= REL_TOL
    gs = g.stats()
    assert gs["ext_rays"] == st["ext_rays"] and gs["shadow_rays"] == st["shadow_rays"]
    g.close()
