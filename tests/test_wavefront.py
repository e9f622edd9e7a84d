"""The wavefront alone: with the tail kernel off, every bounce of every path goes
through the iteration kernels (generate, trace, shade, shadow trace, finish),
however few paths are left.  Each path's colour has to be the oracle's, and the
bits that the tail kernel gives."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL_TOL = 1e-4  # the parity contract of the path tracer
AUTO = 0xFFFFFFFF  # PT_TAIL_AUTO


def rel_err(a, b):
    return np.abs(a - b) / np.maximum(np.maximum(np.abs(a), np.abs(b)), 1e-3)


def scenes(P):
    return {
        "cornell_ref": lambda: (P.cornell_reference(64, 64), 64, 64, dict(rr_depth=10)),
        "cornell_c1": lambda: (P.cornell_c1(64, 64), 64, 64, dict(rr_depth=3)),
        "spheres": lambda: (P.random_spheres(96, 54), 96, 54, dict(rr_depth=10)),
        "zoo": lambda: (P.material_zoo(80, 60), 80, 60, dict(rr_depth=10)),
        "terrain": lambda: (P.heightfield_scene(96, 54, cells=48, env_w=256, env_h=128), 96, 54,
                            dict(rr_depth=10)),
        "moving": lambda: (P.moving_spheres(96, 54), 96, 54, dict(rr_depth=10)),
        "textures": lambda: (P.texture_zoo(81, 63), 81, 63, dict(rr_depth=10)),
    }


NAMES = ["cornell_ref", "cornell_c1", "spheres", "zoo", "terrain", "moving", "textures"]


def wavefront_only(g):
    assert g.lib.pt_set_tail_limit(g.ctx, 0) == 0
    return g


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("slots", [0, 999])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name", NAMES)
def test_every_bounce_equals_oracle(ptgb_mod, oracle_mod, name, mode, slots, order):
    s, w, h, kw = scenes(ptgb_mod)[name]()
    prm = ptgb_mod.GpuRenderer.params(w, h, 1, frame0=3, mode=mode, **kw)
    tail = ptgb_mod.GpuRenderer(s)
    assert tail.lib.pt_set_tail_limit(tail.ctx, 1 << 20) == 0
    ref_tail = tail.render_paths(prm).reshape(-1, 3)
    st = tail.stats()
    assert st["iterations"] == 1                 # one launch took them all
    g = wavefront_only(ptgb_mod.GpuRenderer(s, path_slots=slots, shade_order=order))
    gpu = g.render_paths(prm).reshape(-1, 3)
    sg = g.stats()
    assert np.array_equal(gpu, ref_tail)
    for k in ("paths", "ext_rays", "shadow_rays"):
        assert sg[k] == st[k]
    # one iteration a bounce: in scenes that paths do not leave at once roulette
    # (past rr_depth) ends the longest; and with few slots the chunk is generated
    # over many iterations
    deep = 3 if name == "terrain" else kw["rr_depth"]
    assert sg["iterations"] - 1 > (deep if slots == 0 else w * h // 1000)
    ref = oracle_mod.Oracle(s).render_paths(w, h, 3, np.arange(w * h), mode=mode, **kw)
    assert rel_err(gpu, ref).max() <= REL_TOL
    assert np.mean(np.all(gpu == ref, axis=1)) > 0.999
    g.close()
    tail.close()


@pytest.mark.parametrize("timing", [False, True])
@pytest.mark.parametrize("mode", [0, 1])
def test_batch(ptgb_mod, mode, timing):
    """All scenes in one wavefront, with depth limits and roulette of their own."""
    sc = scenes(ptgb_mod)
    jobs, refs = [], []
    for k, name in enumerate(NAMES):
        s, w, h, kw = sc[name]()
        if name == "zoo":
            kw = dict(max_depth=7)
        g = ptgb_mod.GpuRenderer(s)
        prm = ptgb_mod.GpuRenderer.params(w, h, 1 + k % 3, mode=mode, **kw)
        refs.append(g.render(prm))
        jobs.append((wavefront_only(g), prm, np.zeros((h, w, 4), np.float32)))
    b = ptgb_mod.Batch(path_slots=4096, timing=timing)
    b.render(jobs)
    for (_, _, acc), ref in zip(jobs, refs):
        assert np.array_equal(acc, ref)
    assert b.stats()["iterations"] > 20
    b.close()
    for g, _, _ in jobs:
        g.close()


@pytest.mark.parametrize("slots", [0, 1000])
@pytest.mark.parametrize("name", ["terrain", "zoo"])
def test_guided(ptgb_mod, name, slots):
    """Guided frames: unguided deep bounces in the wavefront or in the tail
    kernel give the same image and train the same weights."""
    w, h = 97, 61
    if name == "terrain":  # whose paths end within the guided bounces
        s = ptgb_mod.heightfield_scene(w, h, cells=48, env_w=128, env_h=64)
    else:
        s = ptgb_mod.material_zoo(w, h)
    got = []
    for limit in (0, AUTO):
        g = ptgb_mod.GpuRenderer(s, path_slots=slots)
        assert g.lib.pt_set_tail_limit(g.ctx, limit) == 0
        g.guide_init(5)
        acc = g.render64(ptgb_mod.GpuRenderer.params(w, h, 3, mode=1, guide=1))
        got.append((acc, *g.guide_state(), g.stats()["iterations"]))
        g.close()
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1]) and got[0][2] == got[1][2]
    assert got[0][3] >= got[1][3] if name == "terrain" else got[0][3] > got[1][3]


@pytest.mark.parametrize("mode", [0, 1])
def test_noalloc_and_host_loop(ptgb_mod, mode):
    torch = pytest.importorskip("torch")
    w, h = 96, 54
    s = ptgb_mod.material_zoo(w, h)
    prm = ptgb_mod.GpuRenderer.params(w, h, 3, mode=mode)
    ref = ptgb_mod.GpuRenderer(s).render(prm)
    g = wavefront_only(ptgb_mod.GpuRenderer(s, path_slots=2000, timing=True, counters=True))
    assert np.array_equal(g.render(prm), ref)
    assert g.stats()["iterations"] > 20
    acc = torch.zeros(h, w, 4, device="cuda")
    rc = g.lib.pt_render_noalloc(g.ctx, ctypes.byref(prm), ctypes.c_void_p(acc.data_ptr()), None)
    assert rc == 0
    torch.cuda.synchronize()
    assert np.array_equal(acc.cpu().numpy(), ref)
    g.close()
