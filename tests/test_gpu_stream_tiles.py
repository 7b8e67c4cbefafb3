"""The plane-streaming kernels against the one-thread-per-cell kernels at the sizes where their
tiles, chunks and rings can go wrong: grids smaller than a tile, ragged last tiles and chunks,
chunks of one plane, odd CPML widths, receivers on never-updated cells, sources next to CPML.

Same arithmetic up to the hardware reciprocal in the harmonic means, so the bounds are those of
test_stream_kernels_match_thread_per_cell_kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(16, 15, 14, 3), (68, 21, 19, 5), (132, 18, 25, 4), (256, 12, 11, 2), (28, 70, 33, 6)]


def _rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


def _batch(torch, grids, nts):
    from elastic_fm_vp_vs_rho_b200 import ShotBatch, configs
    b = ShotBatch()
    for i, (nx, ny, nz, W) in enumerate(grids):
        rng = np.random.default_rng(nx)
        vp = 3000. + 200. * rng.random((ny, nz, nx))
        vs, rho = vp / 1.8, 2000. + 100. * rng.random((ny, nz, nx))
        mu = rho * vs**2
        lam = rho * vp**2 - 2 * mu
        dev = [torch.as_tensor(a.astype(np.float32), device="cuda") for a in (lam, mu, rho)]
        n = nts[i]
        dt, dx = 0.0008, 10.
        rec = [[0, ny // 2, 1], [nx - 1, ny - 1, nz - 1], [W, W, 2], [nx // 2, ny // 2, 3], [nx // 2, ny // 2, 3],
               [nx - W - 1, ny - W - 1, nz - W - 1], [nx // 2 + 1, 2, nz // 2]]
        b.add(nx=nx, ny=ny, nz=nz, lenpml=W, dx=dx, dt=dt, nt=n,
              cpml=configs.cpml_profiles(20., dt, dx, W, 3000., nx, ny, nz), lam=dev[0], mu=dev[1], rho=dev[2],
              wavelet=configs.ricker(25., dt, n) * 1e6, src=[[nx // 2, ny // 2, nz // 2], [W, ny // 2, 4]],
              mt=[[1., .5, -.5, .3, .2, .1], [.4, 1., .2, .1, .6, -.2]], rec=rec)
    return b


def _run(torch, stream, ychunk, rows, pair, grids, nts=(70,)):
    from elastic_fm_vp_vs_rho_b200 import _lib
    b = _batch(torch, grids, nts)
    b.set_option(_lib.EFM_OPT_STREAM_KERNELS, stream)
    b.set_option(_lib.EFM_OPT_YCHUNK, ychunk)
    b.set_option(_lib.EFM_OPT_TILE_ROWS, rows)
    b.set_option(_lib.EFM_OPT_PAIR_LAUNCH, pair)
    mod = b.forward(save_borders=True)
    g, m = b.gradient(mod, model=True, mt=True)
    b.status()
    out = (mod.cpu().numpy(), [b.grad_view(g, i).cpu().numpy() for i in range(len(grids))], m.cpu().numpy())
    b.close()
    return out


SHAPES = pytest.mark.parametrize("ychunk,rows,pair", [(0, 2, 1), (1, 2, 1), (3, 1, 1), (0, 2, 0)])


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g)))
@SHAPES
def test_stream_tiles_match_thread_per_cell_kernels(cuda, grid, ychunk, rows, pair):
    m1, g1, t1 = _run(cuda, 1, ychunk, rows, pair, [grid])
    m2, g2, t2 = _run(cuda, 0, ychunk, rows, pair, [grid])
    assert _rel(m1, m2) < 1e-5
    for i in range(3):
        assert _rel(g1[0][i], g2[0][i]) < 5e-5
    assert _rel(t1, t2) < 2e-5


@SHAPES
def test_stream_tiles_of_an_uneven_batch_equal_separate_runs(cuda, ychunk, rows, pair):
    """Grids of unlike shapes and record lengths share a launch's chunks: bit for bit what each
    gives by itself (with its own tiles and chunk length)."""
    nts = [70 - 13 * i for i in range(len(GRIDS))]
    _, g, _ = _run(cuda, 1, ychunk, rows, pair, GRIDS, nts)
    for i, grid in enumerate(GRIDS):
        _, one, _ = _run(cuda, 1, ychunk, rows, pair, [grid], nts[i:])
        assert np.array_equal(g[i], one[0])


@pytest.mark.parametrize("grids,rows", [([(40, 36, 30, 6)], 1), ([(100, 90, 80, 10)], 2), (GRIDS[:3], 1)], ids=str)
def test_exact_gradient_tile_choice_and_dependent_launches(cuda, grids, rows):
    """Grids that fill the device with 32 x 16 tiles take them, others 32 x 8: bit for bit what that
    option gives, with dependent launches and plain ones.  (The two tiles' kernels are compiled
    apart and may round an operand of a small sum differently.)"""
    from elastic_fm_vp_vs_rho_b200 import _lib
    out = []
    for option, pdl in ((0, 1), (0, 0), (rows, 1), (rows, 0)):
        b = _batch(cuda, grids, [30] * len(grids))
        b.set_option(_lib.EFM_OPT_TILE_ROWS, option)
        b.set_option(_lib.EFM_OPT_PDL, pdl)
        b.set_option(_lib.EFM_OPT_CHECKPOINT_EVERY, 8)
        mod = b.forward(checkpoints=True)
        g, m = b.gradient(mod, exact=True, mt=True)
        b.status()
        out.append((g.cpu().numpy(), m.cpu().numpy()))
        b.close()
    for g, m in out[1:]:
        assert np.array_equal(g, out[0][0]) and np.array_equal(m, out[0][1])
