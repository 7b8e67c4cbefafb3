"""A tuned batch's exact gradient chooses its own tiles and chunks.

The tuner times the stencil passes; what it sets for them used to pick the exact adjoint's tiles as
well: 32 x 16 on grids that they cannot fill (29.3 ms a 48x48x40 gradient, 27.2 with 32 x 8), 32 x 8
on large ones (106 ms at 128x128x96, 85)."""
import pytest

from test_gpu_stream_tiles import _batch


def test_apply_leaves_the_exact_adjoint_to_itself():
    from elastic_fm_vp_vs_rho_b200 import _lib, autotune

    class Batch:
        options = {}

        def set_option(self, option, value):
            self.options[option] = value

    autotune.apply(Batch(), {"rows": 2, "ring": 4, "ychunk": 5})
    assert Batch.options == {_lib.EFM_OPT_TILE_ROWS: 2, _lib.EFM_OPT_RING_DEPTH: 4, _lib.EFM_OPT_YCHUNK: 5,
                             _lib.EFM_OPT_EXACT_SHAPE: 1}


@pytest.mark.gpu
@pytest.mark.parametrize("grid,choice", [((48, 48, 40, 8), (2, 4, 16)), ((128, 128, 96, 10), (1, 6, 8))], ids=str)
def test_tuned_exact_gradient_is_the_untuned_one(cuda, grid, choice):
    """The same bits (the two tiles' results differ in a few cells' last ones) within 6 % of the time."""
    from elastic_fm_vp_vs_rho_b200 import autotune
    out, us = [], []
    for tuned in (False, True):
        b = _batch(cuda, [grid], [60])
        if tuned:
            autotune.apply(b, dict(zip(("rows", "ring", "ychunk"), choice)))
        mod = b.forward(checkpoints=True)
        g, m = b.gradient(mod, exact=True, mt=True)
        out.append((g.clone(), m.clone()))
        times = []
        for _ in range(6):
            b.forward(checkpoints=True, out=mod)
            e0, e1 = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            e0.record()
            b.gradient(mod, exact=True, mt=True)
            e1.record()
            cuda.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        us.append(min(times))
        b.status()
        b.close()
    assert cuda.equal(out[0][0], out[1][0]) and cuda.equal(out[0][1], out[1][1])
    assert us[1] <= 1.06 * us[0]
