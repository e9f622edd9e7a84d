"""First-hit queries answered through host memory (up to 16384 rays) and past
that size: ids and distances equal the oracle's, into host arrays (unaligned
ones too) and into device memory."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["cornell", "zoo"])
@pytest.mark.parametrize("w,h", [(1, 1), (33, 1), (128, 128), (129, 128)])
def test_first_hit_sizes(ptgb_mod, oracle_mod, name, w, h):
    torch = pytest.importorskip("torch")
    s = ptgb_mod.cornell_c1(w, h) if name == "cornell" else ptgb_mod.material_zoo(w, h)
    g = ptgb_mod.GpuRenderer(s)
    ref = oracle_mod.Oracle(s).first_hits(w, h, 2)
    for a, b in zip(g.first_hits(w, h, 2), ref):
        assert np.array_equal(a, b)
    n = 4 * w * h
    host = [np.zeros(n + 1, np.uint8) for _ in range(3)]       # byte offset 1
    p = [ctypes.c_void_p(a.ctypes.data + 1) for a in host]
    assert g.lib.pt_trace_first_hits(g.ctx, w, h, 2, *p, None) == 0
    for a, b in zip(host, ref):
        assert a[1:].tobytes() == np.ascontiguousarray(b).tobytes()
    dev = [torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(a.data_ptr()) for a in dev]
    assert g.lib.pt_trace_first_hits(g.ctx, w, h, 2, *p, None) == 0
    for a, b in zip(dev, ref):
        assert a.cpu().numpy().tobytes() == np.ascontiguousarray(b).tobytes()
    g.close()
