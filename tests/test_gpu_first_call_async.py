"""The first forward and gradient of a batch are queued behind the stream's work, not waited for.

Allocations and tables are made while a kernel that takes about 0.2 s runs on the stream; the calls
return long before it ends (5 ms on a batch not run before), with every block size."""
import time

import pytest

from test_gpu_stream_tiles import _batch

pytestmark = pytest.mark.gpu

CYCLES = 400_000_000  # about 0.2 s of the device


@pytest.mark.parametrize("rows", [0, 1])
def test_first_calls_return_while_the_stream_is_busy(cuda, rows):
    from elastic_fm_vp_vs_rho_b200 import _lib
    grids, nts = [(48, 40, 36, 6), (64, 30, 28, 5)], [20, 16]

    def fresh():
        b = _batch(cuda, grids, nts)
        b.set_option(_lib.EFM_OPT_TILE_ROWS, rows)
        cuda.cuda.synchronize()
        return b

    stream = cuda.cuda.Stream()
    waited = []
    for attempt in range(3):  # (the first one loads the kernels, which waits for the device)
        b = fresh()
        with cuda.cuda.stream(stream):
            cuda.cuda._sleep(CYCLES)
            end = cuda.cuda.Event()
            end.record()
            t = time.perf_counter()
            mod = b.forward(save_borders=True)
            b.gradient(mod, model=True, mt=True)
            waited.append((time.perf_counter() - t, end.query()))
        stream.synchronize()
        b.status()
        b.close()
    seconds, done = min(waited[1:])
    assert not done, f"the calls waited for the stream: {seconds:.3f} s"
