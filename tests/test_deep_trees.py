"""Triangle meshes on which clustering chains (coincident triangles, nested
sizes, areas past the range of a float): the committed tree is no deeper than
the treelet builder's, pt_commit takes it at every node width, and rays find
what the CPU oracle finds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mesh(kind, n):
    r = np.random.RandomState(n)
    if kind == "same":
        return np.repeat(r.uniform(-0.8, 0.8, (1, 3, 3)), n, 0)
    if kind == "nested":
        return r.uniform(-0.5, 0.5, (n, 3, 3)) * 1.01 ** (np.arange(n) % 3000)[:, None, None] * 1e-6
    return r.uniform(0, 1e20, (n, 1, 3)) + r.uniform(-5e18, 5e18, (n, 3, 3))  # "huge"


# (kind, triangles, node width): deepest tree allowed.  Clustering alone makes
# 25, 157, 205, 43, 117 and 155 levels, and a trace block's stacks hold 124.
@pytest.mark.parametrize("builder", [0, 2])
@pytest.mark.parametrize("kind,n,width,deepest", [("same", 5000, 8, 14), ("same", 5000, 2, 60),
                                                  ("same", 65536, 2, 90), ("nested", 5000, 8, 40),
                                                  ("huge", 5000, 8, 20), ("huge", 65536, 8, 24)])
def test_commit(ptgb_mod, oracle_mod, kind, n, width, deepest, builder):
    w, h = 48, 36
    s = ptgb_mod.Scene()
    v = mesh(kind, n).astype(np.float32).reshape(-1, 3)
    s.mesh(v, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3), s.lambertian((0.7, 0.6, 0.5)))
    s.miss_gradient((1.0, 1.0, 1.0), (0.5, 0.7, 1.0))
    s.set_camera((0.3, 0.4, 3.0), (0.0, 0.0, 0.0), (0, 1, 0), 60.0, w / h, 0.0, 2.0)
    g, o = ptgb_mod.GpuRenderer(s, builder=builder, bvh_width=width), oracle_mod.Oracle(s)
    assert g.stats()["bvh_depth"] <= deepest
    for a, b in zip(g.first_hits(w, h, 1)[:2], o.first_hits(w, h, 1)[:2]):
        assert np.array_equal(a, b)
    gpu = g.render_paths(ptgb_mod.GpuRenderer.params(w, h, 1, frame0=2, max_depth=4)).reshape(-1, 3)
    assert np.array_equal(gpu, o.render_paths(w, h, 2, np.arange(w * h), max_depth=4))
    g.close()
