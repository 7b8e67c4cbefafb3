"""The illumination of a cell is the float32 sum over the steps of vz^2 + (vx^2 + vy^2), the squares
of x and z fused into the sums: exactly, from the velocities recorded at the cell."""
from fractions import Fraction

import numpy as np
import pytest

from test_gpu_stream_tiles import _batch

pytestmark = pytest.mark.gpu


def _fma(a, b, c):
    return np.float32(float(Fraction(float(a)) * Fraction(float(b)) + Fraction(float(c))))


@pytest.mark.parametrize("rows", [2, 1])
def test_illumination_from_recorded_velocities(cuda, rows):
    from elastic_fm_vp_vs_rho_b200 import _lib
    b = _batch(cuda, [(36, 27, 22, 5)], [50])
    b.set_option(_lib.EFM_OPT_TILE_ROWS, rows)
    illum = cuda.zeros(b.illum_size, device="cuda")
    v = b.gather_view(b.forward(illum=illum), 0).cpu().numpy()
    vol = b.illum_view(illum, 0).cpu().numpy()
    rec = b.specs[0]["rec"]
    b.status()
    checked = 0
    for r, (x, y, z) in enumerate(rec):
        if not (2 <= x < 34 and 2 <= y < 25 and 2 <= z < 20):
            continue
        e = np.float32(0)
        for vx, vy, vz in v[:, :, r].T:
            e = np.float32(e + _fma(vz, vz, _fma(vx, vx, np.float32(vy * vy))))
        assert vol[y, z, x] == e
        checked += e > 0
    assert checked >= 3
    b.close()
