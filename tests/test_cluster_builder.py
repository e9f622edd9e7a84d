"""The clustered GPU BVH of triangle meshes against the CPU oracle: sizes
around the cluster and warp limits, coincident triangles (equal codes and
areas), and a closed room, whose walls lie on node boundaries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def soup(n, kind):
    r = np.random.RandomState(n)
    c = r.uniform(-1, 1, (n, 1, 3)) if kind != "same" else np.zeros((n, 1, 3))
    d = r.uniform(-0.4, 0.4, (1 if kind == "same" else n, 3, 3))
    return (c + d).astype(np.float32).reshape(-1, 3)


def scene_of(ptgb, verts, w, h, eye):
    s = ptgb.Scene()
    m = s.lambertian((0.7, 0.6, 0.5))
    s.mesh(verts, np.arange(len(verts), dtype=np.uint32).reshape(-1, 3), m)
    s.miss_gradient((1.0, 1.0, 1.0), (0.5, 0.7, 1.0))
    s.set_camera(eye, (0.0, 0.0, 0.0), (0, 1, 0), 60.0, w / h, 0.0, 2.0)
    return s


def check(ptgb, oracle, s, w, h, **kw):
    g, o = ptgb.GpuRenderer(s, builder=2, **kw), oracle.Oracle(s)
    for a, b in zip(g.first_hits(w, h, 1)[:2], o.first_hits(w, h, 1)[:2]):
        assert np.array_equal(a, b)
    gpu = g.render_paths(ptgb.GpuRenderer.params(w, h, 1, frame0=2)).reshape(-1, 3)
    assert np.array_equal(gpu, o.render_paths(w, h, 2, np.arange(w * h)))
    g.close()


@pytest.mark.parametrize("kind", ["random", "same"])
@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 32, 33, 255, 257, 5000])
def test_sizes(ptgb_mod, oracle_mod, n, kind):
    check(ptgb_mod, oracle_mod, scene_of(ptgb_mod, soup(n, kind), 48, 36, (0.3, 0.4, 3.0)), 48, 36)


@pytest.mark.parametrize("width", [2, 3, 7])
def test_widths(ptgb_mod, oracle_mod, width):
    s = scene_of(ptgb_mod, soup(700, "random"), 48, 36, (0.3, 0.4, 3.0))
    check(ptgb_mod, oracle_mod, s, 48, 36, bvh_width=width)


def test_closed_room(ptgb_mod, oracle_mod):
    k = 13                                      # walls of 13 x 13 cells, the camera inside
    i, j = np.meshgrid(np.arange(k), np.arange(k), indexing="ij")
    a, b = i.reshape(-1) / k * 2 - 1, j.reshape(-1) / k * 2 - 1
    e = 2.0 / k
    tri = np.stack([np.stack([a, b], -1), np.stack([a + e, b], -1), np.stack([a, b + e], -1),
                    np.stack([a + e, b], -1), np.stack([a + e, b + e], -1),
                    np.stack([a, b + e], -1)], 1).reshape(-1, 2)
    walls = []
    for axis in range(3):
        for side in (-1.02, 1.02):
            v = np.insert(1.02 * tri, axis, side, axis=1)
            walls.append(v)
    verts = np.concatenate(walls).astype(np.float32)
    check(ptgb_mod, oracle_mod, scene_of(ptgb_mod, verts, 160, 120, (0.2, 0.3, 0.9)), 160, 120)
