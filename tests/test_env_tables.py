"""The environment's CDF search tables (a search starts between the entries of
neighbouring table positions) against the CPU oracle's whole-CDF searches:
odd and tiny sizes, rows without light, one texel that holds nearly all of
it, and a total that is not finite (then the tables are not used)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL_TOL = 1e-4  # the parity contract of the path tracer


def env_of(kind, w, h):
    r = np.random.RandomState(w * 1000 + h)
    env = r.uniform(0.0, 1.0, (h, w, 4)).astype(np.float32)
    if kind == "dark_rows":
        env[::2] = 0.0
        env[h // 2, :, :3] = 0.25
    elif kind == "spike":
        env[..., :3] *= 1e-6
        env[h // 3, w // 2, :3] = 5e4
    elif kind == "infinite":
        env[h // 3, w // 2, 0] = np.inf
    return env


@pytest.mark.parametrize("kind,w,h", [("flat", 1, 1), ("flat", 3, 5), ("flat", 64, 32),
                                      ("dark_rows", 37, 19), ("spike", 129, 65), ("spike", 255, 7),
                                      ("infinite", 33, 17)])
def test_env_search_tables(ptgb_mod, oracle_mod, kind, w, h):
    s = ptgb_mod.material_zoo(64, 48)
    s.miss_env(env_of(kind, w, h), spherical=True)
    g, o = ptgb_mod.GpuRenderer(s), oracle_mod.Oracle(s)
    prm = ptgb_mod.GpuRenderer.params(64, 48, 1, frame0=1, mode=1)
    gpu = g.render_paths(prm).reshape(-1, 3)
    ref = o.render_paths(64, 48, 1, np.arange(64 * 48), mode=1)
    fine = np.isfinite(ref)
    assert np.array_equal(fine, np.isfinite(gpu))
    gpu, ref = gpu[fine], ref[fine]
    err = np.abs(gpu - ref) / np.maximum(np.maximum(np.abs(gpu), np.abs(ref)), 1e-3)
    assert err.max() <= REL_TOL
    g.close()
