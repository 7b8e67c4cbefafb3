"""efm_kernel_time after a call whose waits ran out: the launches do all their work again.

A block that gives up leaves numbers of the launch's chunk counter unfetched, and every streaming
launch starts from that counter.  With chunks of one plane and a one-poll limit each block of the
four launches takes two numbers of 3472: two thirds are gone when the timing starts, and its first
launch would do a third of the work.
"""
import ctypes

import pytest

from test_gpu_stream_tiles import _batch

pytestmark = pytest.mark.gpu


def test_timed_launch_does_all_chunks_after_a_timeout(cuda):
    from elastic_fm_vp_vs_rho_b200 import _lib
    b = _batch(cuda, [(128, 128, 96, 10)], [2])
    b.set_option(_lib.EFM_OPT_YCHUNK, 1)

    def stress_us(reps):
        ms = ctypes.c_double()
        _lib.check(_lib.load().efm_kernel_time(b._ctx, 0, reps, 0, ctypes.byref(ms), _lib.stream_ptr()))
        return 1e3 * ms.value

    b.forward()
    full = min(stress_us(1) for _ in range(8))
    b.status()
    b.set_option(_lib.EFM_OPT_WAIT_LIMIT, 1)
    b.forward()
    with pytest.raises(_lib.EfmError):
        b.status()
    b.set_option(_lib.EFM_OPT_WAIT_LIMIT, 0)
    after = stress_us(1)
    b.status()
    assert after > 0.8 * full
    b.close()
