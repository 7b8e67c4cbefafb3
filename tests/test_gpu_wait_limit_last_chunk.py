"""Consumers that give up after the producer has issued its last load: the block still waits for it.

With chunks of one plane a block has two slots to fill, fewer than its barriers, so its producer
issues everything and writes the end mark without waiting for a consumer; a short limit then makes
the consumers give up on those loads.  Limits around a load's latency give up in some blocks and
slots and not in others.  The call completes, the status is a timeout (always for one poll) or
success, and the next calls with the default limit are bit-identical to ones before.  Every wait is
bounded and every load completes on its own.
"""
import pytest

from test_gpu_stream_tiles import _batch

pytestmark = pytest.mark.gpu


def _run(b, gathers):
    mod = b.forward(save_borders=True)
    g, m = b.gradient(gathers if gathers is not None else mod, model=True, mt=True)
    return mod, g, m


@pytest.mark.parametrize("rows,ring", [(2, 4), (1, 4), (1, 6)])
@pytest.mark.parametrize("ychunk", [1, 3])
def test_consumers_that_give_up_on_the_last_loads(cuda, rows, ring, ychunk):
    from elastic_fm_vp_vs_rho_b200 import _lib
    b = _batch(cuda, [(40, 26, 20, 4), (16, 15, 14, 3)], [12, 9])
    b.set_option(_lib.EFM_OPT_TILE_ROWS, rows)
    b.set_option(_lib.EFM_OPT_RING_DEPTH, ring)
    b.set_option(_lib.EFM_OPT_YCHUNK, ychunk)
    ref = _run(b, None)
    b.status()
    timeouts = []
    for limit in (1, 8, 40, 200):
        b.set_option(_lib.EFM_OPT_WAIT_LIMIT, limit)
        b.forward(save_borders=True)
        try:
            b.status()
            timeouts.append(False)
        except _lib.EfmError as e:
            assert e.code == _lib.EFM_ERR_TIMEOUT
            timeouts.append(True)
        b.set_option(_lib.EFM_OPT_WAIT_LIMIT, 0)
        b.forward(save_borders=True)
        b.status()
        b.set_option(_lib.EFM_OPT_WAIT_LIMIT, limit)
        b.gradient(ref[0], model=True, mt=True)
        try:
            b.status()
        except _lib.EfmError as e:
            assert e.code == _lib.EFM_ERR_TIMEOUT
        b.set_option(_lib.EFM_OPT_WAIT_LIMIT, 0)
        for a, r in zip(_run(b, ref[0]), ref):
            assert cuda.equal(a, r)
        b.status()
    assert timeouts[0]
    b.close()
