"""Host-built trees whose wide nodes are chosen by the cost of their quantised
boxes: structure and containment (host code), and renders against the CPU
oracle for scenes on a ground that dwarfs everything else."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "optix-path-tracer_gb300", "csrc")


def test_fit_tree_boxes(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "fit_tree")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", CSRC, os.path.join(HERE, "fit_tree_driver.cpp"),
                    os.path.join(CSRC, "bvh_host.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    lines = out.stdout.strip().splitlines()
    assert out.returncode == 0 and lines[-1] == "ALL PASS", [l for l in lines if "FAIL" in l]
    assert sum(l.startswith("PASS ") for l in lines) == 4 * 7 * 8


# one node, the first sizes past it, ordinary ones; with a light quad above
# (moving) and without; triangles on both sides of the GPU builder's 512
@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("kind,size", [("spheres", 0), ("spheres", 1), ("spheres", 2), ("spheres", 6),
                                       ("moving", 1), ("moving", 4), ("terrain", 15), ("terrain", 16),
                                       ("nested", 511), ("nested", 600)])
def test_fit_tree_renders(ptgb_mod, oracle_mod, kind, size, mode):
    w, h = 96, 61
    if kind == "spheres":
        s = ptgb_mod.random_spheres(w, h, 3, size)
    elif kind == "moving":
        s = ptgb_mod.moving_spheres(w, h, 3, size)
    elif kind == "nested":  # triangles from 1 to 5e7 in size around one point: deep trees
        s = ptgb_mod.Scene()
        s.miss_gradient((1.0, 1.0, 1.0), (0.5, 0.7, 1.0))
        k = np.arange(size)
        a = 2.4 * k[:, None] + np.array([0.0, 0.4, 0.2])
        r = 1.03 ** k[:, None] * np.array([1.0, 1.0, 1.1])
        v = np.stack([r * np.cos(a), r * np.sin(a), r * np.array([-1.0, -0.9, -1.2])], axis=2)
        s.mesh(v.reshape(-1, 3).astype(np.float32), np.arange(3 * size, dtype=np.uint32),
               s.lambertian((0.6, 0.5, 0.4)))
        s.set_camera((0, 0, 0), (0, 0, -1), (0, 1, 0), 100.0, w / h, 0.0, 1.0)
    else:
        s = ptgb_mod.heightfield_scene(w, h, cells=size, seed=3, env_w=64, env_h=32)
    g, o = ptgb_mod.GpuRenderer(s), oracle_mod.Oracle(s)
    for a, b in zip(g.first_hits(w, h, 1), o.first_hits(w, h, 1)):
        assert np.array_equal(a, b)
    gpu = g.render_paths(ptgb_mod.GpuRenderer.params(w, h, 1, frame0=2, mode=mode)).reshape(-1, 3)
    assert np.array_equal(gpu, o.render_paths(w, h, 2, np.arange(w * h), mode=mode))
    g.close()


@pytest.mark.gpu
def test_fit_tree_fetches(ptgb_mod):
    """488 spheres on a ground sphere of radius 1000 (whose grid step under the
    root is 8): fewer than five node fetches a ray (8.6 when the root held the
    small spheres' nodes itself)."""
    s = ptgb_mod.random_spheres(320, 180)
    g = ptgb_mod.GpuRenderer(s, counters=True)
    g.render(ptgb_mod.GpuRenderer.params(320, 180, 1))
    st = g.stats()
    assert st["node_fetches"] < 5 * st["ext_rays"]
    g.close()
