"""Device memory of the path state: the shading lists (32 bytes a slot) are there
only for scenes shaded by lists, and a context keeps one copy of its normals."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def used(torch):
    torch.cuda.synchronize()
    return -torch.cuda.mem_get_info()[0]


def growth(torch, ptgb, order, batch):
    """Bytes that the first render of a context (or batch) of 4 Mi slots takes."""
    w = h = 160
    s = ptgb.material_zoo(w, h)
    g = ptgb.GpuRenderer(s, path_slots=0 if batch else 4 * MIB, shade_order=order)
    b = ptgb.Batch(path_slots=4 * MIB, shade_order=order) if batch else None
    acc = torch.zeros(h, w, 4, device="cuda")
    prm = ptgb.GpuRenderer.params(w, h, 1, mode=1)
    before = used(torch)
    if batch:
        b.render([(g, prm, acc.data_ptr())])
    else:
        g.render(prm, acc.data_ptr())
    grown = used(torch) - before
    if batch:
        b.close()
    g.close()
    return grown


@pytest.mark.parametrize("batch", [False, True])
def test_lists_only_where_used(ptgb_mod, batch):
    torch = pytest.importorskip("torch")
    growth(torch, ptgb_mod, 1, batch)            # what is allocated once per process
    lists, order = growth(torch, ptgb_mod, 1, batch), growth(torch, ptgb_mod, 2, batch)
    # 32 bytes x 4 Mi slots, in allocations of 2 MiB; path state of 304 bytes a slot
    assert abs(lists - order - 128 * MIB) <= 16 * MIB
    assert 304 * 4 * MIB <= order <= 304 * 4 * MIB + 32 * MIB


def test_one_copy_of_normals(ptgb_mod):
    """A commit keeps 16 bytes of normals a vertex; the caller's 12 go through
    the scratch of the sky's sampling tables."""
    torch = pytest.importorskip("torch")
    n, w, h = 4 * MIB, 4096, 2048                # 12 bytes a vertex are less than 8 a texel

    def commit():
        verts = np.random.default_rng(0).random((n, 3), dtype=np.float32)
        s = ptgb_mod.Scene()
        s.mesh(verts, np.arange(3000, dtype=np.uint32).reshape(-1, 3), s.lambertian((0.5, 0.5, 0.5)),
               normals=verts)
        s.miss_env(np.ones((h, w, 4), np.float32), spherical=True)
        s.set_camera((0, 0, 3), (0, 0, 0), (0, 1, 0), 40.0, 1.0, 0.0, 3.0)
        before = used(torch)
        g = ptgb_mod.GpuRenderer(s)
        grown = used(torch) - before
        g.close()
        return grown

    commit()                                     # what is allocated once per process
    sky = 16 * w * h + 8 * w * h + 4 * (w + 1) * h + 2 * (w + 1) * h  # texels, scratch, CDFs, search tables
    assert abs(commit() - (sky + 16 * n + 8 * n)) <= 24 * MIB  # normals and uvs; the rest is small
