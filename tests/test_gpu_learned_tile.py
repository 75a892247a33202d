"""The training tile (tracer_set_cells_per_block) changed after the learned flux
was set: the loss's partial sums follow the number of blocks."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [0, 48])
@pytest.mark.parametrize("fct", [0, 1])
def test_training_step_after_the_tile_changed(api, fct, first):
    """The tile at which the learned flux is set (the default, or one given before), 32 cells per block (16 times the blocks), 576 and the default
    again: one loss and one gradient.  The loss is an FP64 sum of at most 33 x 33 x
    11 terms, reordered (12,000 x 2^-53 = 1.3e-12 relative); the gradient's order of
    FP32 additions over at most 296 blocks is never fixed (296 x 2^-24 = 1.8e-5)."""
    from fesom2_tracer_dwarf_b200.learned import coarse_setup, init_params
    from fesom2_tracer_dwarf_b200.workloads import cfl_dt
    nx, nl = 33, 12
    uv, w, amp, _ = coarse_setup(api, nx, nl, 6)
    dt = cfl_dt(api, nx, nx, nl, uv, w)
    T = np.asfortranarray(api.synth_tracer(seed=4, kind=2))
    target = np.asfortranarray(T + 0.05 * np.sin(np.arange(T.size)).reshape(T.shape, order="F"))
    api.set_precision("fp32")
    api.allocate_tracers(1)
    api.set_scheme(1, "MUSCL", "PPM", "FCT")
    api.set_velocity(uv, w)
    api.set_ab_refresh(True)
    p = init_params(3)
    p[5248:5312] = np.random.default_rng(2).standard_normal(64).astype(np.float32) * 0.3
    got = []
    for cells in (first, 32, 576, 0):
        api.set_cells_per_block(cells)
        if not got:
            assert api.lib.tracer_learn_set(p.ctypes.data, 0) == 0
        loss = ctypes.c_double()
        assert api.lib.tracer_learn_step(T.ctypes.data, target.ctypes.data, dt, 0.0, 1, fct, ctypes.byref(loss)) == 0
        g = np.zeros_like(p)
        assert api.lib.tracer_learn_grad(g.ctypes.data) == 0
        got.append((loss.value, g))
    l0, g0 = got[0]
    assert l0 > 0.0 and np.linalg.norm(g0) > 0.0
    for loss, g in got[1:]:
        assert abs(loss - l0) <= 2e-12 * l0
        assert np.linalg.norm(g - g0) <= 2e-5 * np.linalg.norm(g0)
