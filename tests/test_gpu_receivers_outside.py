"""Receivers on cells the stencil never updates (they record zeros and take the adjoint source).

The velocity pass covers the updated cells and is extended in y and z as far as such receivers
reach: against the thread-per-cell kernels for every face and for corners (bounds of
test_stream_tiles_match_thread_per_cell_kernels), and by the clock a receiver line on z = 0 costs
what one on z = 2 does (a pass over the whole grid took 9 % longer here)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID = (36, 27, 22, 5)
FACES = {"z0": [[9, 9, 0], [12, 20, 1]], "z1": [[9, 9, 21], [30, 13, 20]], "y0": [[9, 0, 9], [20, 1, 5]],
         "y1": [[9, 26, 9], [20, 25, 15]], "x": [[0, 9, 9], [1, 13, 9], [35, 9, 9], [34, 13, 2]],
         "corners": [[0, 0, 0], [35, 26, 21]], "y0z1": [[18, 1, 20]]}


def _batch(torch, nx, ny, nz, W, nt, rec):
    from elastic_fm_vp_vs_rho_b200 import ShotBatch, configs
    vp = 3000. + 200. * torch.rand((ny, nz, nx), generator=torch.Generator().manual_seed(1))
    vp = vp.cuda()
    mu = 2000. * (vp / 1.8)**2
    b = ShotBatch()
    b.add(nx=nx, ny=ny, nz=nz, lenpml=W, dx=10., dt=0.0008, nt=nt,
          cpml=configs.cpml_profiles(20., 0.0008, 10., W, 3000., nx, ny, nz), lam=2000. * vp**2 - 2. * mu, mu=mu,
          rho=torch.full_like(vp, 2000.), wavelet=1e6 * configs.ricker(25., 0.0008, nt),
          src=[[nx // 2, ny // 2, nz // 2]], mt=[[1., .5, -.5, .3, .2, .1]], rec=rec)
    return b


@pytest.mark.parametrize("face", list(FACES))
@pytest.mark.parametrize("rows,ychunk", [(2, 0), (1, 3)])
def test_receivers_outside_match_thread_per_cell_kernels(cuda, face, rows, ychunk):
    from elastic_fm_vp_vs_rho_b200 import _lib
    nt, inside = 60, [[20, 14, 4], [7, 20, 12]]
    out = []
    for stream in (1, 0):
        b = _batch(cuda, *GRID, nt, FACES[face] + inside)
        b.set_option(_lib.EFM_OPT_STREAM_KERNELS, stream)
        b.set_option(_lib.EFM_OPT_TILE_ROWS, rows)
        b.set_option(_lib.EFM_OPT_YCHUNK, ychunk)
        mod = b.forward(save_borders=True)
        assert not mod.view(3, nt, -1)[:, :, :len(FACES[face])].any()
        # adjoint sources at every receiver, the outer ones included
        res = cuda.linspace(-1, 1, mod.numel(), device="cuda") * mod.abs().max()
        g, m = b.gradient(res, model=True, mt=True)
        b.status()
        out.append([a.cpu().numpy() for a in (mod, g, m)])
        b.close()
    for a, ref, bound in zip(out[0], out[1], (1e-5, 5e-5, 2e-5)):
        assert np.abs(a - ref).max() <= bound * np.abs(ref).max()


def test_surface_receivers_do_not_extend_the_pass(cuda):
    def forward_us(z):
        b = _batch(cuda, 64, 64, 64, 10, 100, [[x, 32, z] for x in range(10, 54, 4)])
        out = b.forward()
        times = []
        for _ in range(6):
            e0, e1 = cuda.cuda.Event(enable_timing=True), cuda.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(4):
                b.forward(out=out)
            e1.record()
            cuda.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        b.close()
        return min(times)

    assert forward_us(0) <= 1.06 * forward_us(2)
