"""A render that fails (here: an iteration bound below what it needs) leaves a
host accumulator as it was, and a device accumulator and the guide as after the
last complete chunk of frames; the context then renders as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 160, 130                                  # past the size that needs no wavefront


def fails(ptgb, g, call):
    with pytest.raises(ptgb.PtError) as e:
        call()
    assert e.value.code == -4                    # PT_ETIMEOUT


# host arrays are copied to before or after the flags are known, by their size
@pytest.mark.parametrize("w,h,spp", [(W, H, 2), (520, 520, 1)])
@pytest.mark.parametrize("timing", [False, True])
@pytest.mark.parametrize("mode", [0, 1])
def test_accumulators_keep_their_values(ptgb_mod, mode, timing, w, h, spp):
    torch = pytest.importorskip("torch")
    g = ptgb_mod.GpuRenderer(ptgb_mod.material_zoo(w, h), path_slots=1000, timing=timing)
    assert g.lib.pt_set_tail_limit(g.ctx, 0) == 0
    prm = ptgb_mod.GpuRenderer.params(w, h, spp, frame0=3, mode=mode)
    first = ptgb_mod.GpuRenderer.params(w, h, spp, mode=mode)  # which starts from zeros
    start = np.random.default_rng(1).random((h, w, 4))
    ref = g.render(prm, start.astype(np.float32))
    ref64 = g.render64(prm, start.copy())
    paths = g.render_paths(prm)
    assert g.lib.pt_set_iteration_limit(g.ctx, 1) == 0
    for dtype, call in ((np.float32, g.render), (np.float64, g.render64)):
        acc = start.astype(dtype)
        fails(ptgb_mod, g, lambda: call(prm, acc))
        fails(ptgb_mod, g, lambda: call(first, acc))
        assert np.array_equal(acc, start.astype(dtype))
        dev = torch.from_numpy(start.astype(dtype)).cuda()
        fails(ptgb_mod, g, lambda: call(prm, dev.data_ptr()))
        assert np.array_equal(dev.cpu().numpy(), start.astype(dtype))
    out = np.full((h, w, 3), 5.0, np.float32)
    fails(ptgb_mod, g, lambda: g.render_paths(prm, out))
    assert np.all(out == 5.0)
    assert g.lib.pt_set_iteration_limit(g.ctx, 0) == 0
    assert np.array_equal(g.render(prm, start.astype(np.float32)), ref)
    assert np.array_equal(g.render64(prm, start.copy()), ref64)
    assert np.array_equal(g.render_paths(prm), paths)
    g.close()


def test_batch_keeps_accumulators(ptgb_mod):
    torch = pytest.importorskip("torch")
    g = ptgb_mod.GpuRenderer(ptgb_mod.material_zoo(W, H))
    b = ptgb_mod.Batch(path_slots=1024)
    prm = ptgb_mod.GpuRenderer.params(W, H, 2, frame0=1, mode=1)
    dev = torch.full((H, W, 4), 2.0, device="cuda")
    ref = dev.clone()
    b.render([(g, prm, ref.data_ptr())])
    assert g.lib.pt_set_iteration_limit(g.ctx, 1) == 0
    fails(ptgb_mod, b, lambda: b.render([(g, prm, dev.data_ptr())]))
    assert bool((dev == 2.0).all())
    assert g.lib.pt_set_iteration_limit(g.ctx, 0) == 0
    b.render([(g, prm, dev.data_ptr())])
    assert bool((dev == ref).all())
    b.close()
    g.close()


def test_guide_keeps_the_complete_frames(ptgb_mod):
    """Of two frames the second needs more iterations than the bound: the
    accumulator and the guide are those of the first alone."""
    torch = pytest.importorskip("torch")
    g = ptgb_mod.GpuRenderer(ptgb_mod.material_zoo(W, H), path_slots=1000)
    g.guide_init(3)

    def frames(f, spp, acc):
        g.render(ptgb_mod.GpuRenderer.params(W, H, spp, frame0=f, mode=1, guide=1), acc.data_ptr())

    states, accs, iters = [g.guide_state()], [], []
    for f in range(1, 12):
        acc = torch.zeros(H, W, 4, device="cuda")
        frames(f, 1, acc)
        states.append(g.guide_state())
        accs.append(acc)
        iters.append(g.stats()["iterations"] - 1)  # without the pass over the last paths
    k = next(k for k in range(len(iters) - 1) if iters[k + 1] > iters[k])
    g.guide_set_state(*states[k])
    assert g.lib.pt_set_iteration_limit(g.ctx, iters[k] + 1) == 0
    acc = torch.zeros(H, W, 4, device="cuda")
    fails(ptgb_mod, g, lambda: frames(k + 1, 2, acc))
    w, step = g.guide_state()
    assert step == states[k + 1][1] and np.array_equal(w, states[k + 1][0])
    assert bool((acc == accs[k]).all())
    assert g.lib.pt_set_iteration_limit(g.ctx, 0) == 0
    frames(k + 2, 1, acc)                        # and it goes on from there
    assert bool((acc == accs[k] + accs[k + 1]).all())
    w, step = g.guide_state()
    assert step == states[k + 2][1] and np.array_equal(w, states[k + 2][0])
    g.close()
