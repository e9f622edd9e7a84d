"""Shading by the lists that the trace kernel fills (one per miss / material
type): wavefronts smaller than a warp chunk and list lengths around its
multiples give the path order's image bit for bit, and every ray once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("slots", [33, 64, 4097])
def test_lists_equal_path_order(ptgb_mod, oracle_mod, slots, mode):
    w, h = 129, 129                              # past the size that needs no wavefront
    s = ptgb_mod.material_zoo(w, h)
    prm = ptgb_mod.GpuRenderer.params(w, h, 1, mode=mode)
    lists = ptgb_mod.GpuRenderer(s, path_slots=slots, shade_order=1)
    order = ptgb_mod.GpuRenderer(s, path_slots=slots, shade_order=2)
    a = lists.render(prm)
    assert np.array_equal(a, order.render(prm))
    _, st = oracle_mod.Oracle(s).render(w, h, 1, mode=mode)
    got = lists.stats()
    assert got["ext_rays"] == st["ext_rays"] and got["shadow_rays"] == st["shadow_rays"]
    lists.close()
    order.close()
