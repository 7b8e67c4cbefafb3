"""Unpaired gradient launches take chunks of their own length, not the pair's.

The two differ where a pass alone fills whole rounds of blocks with a chunk that leaves the pair a
part of one.  By the clock, since every chunk length gives the same bits: the rule may miss the best
of three lengths set by hand by 14 %; the pair's chunks miss it by more than 20 %."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NT = 60


def _batch(torch, nx, ny, nz, W):
    from elastic_fm_vp_vs_rho_b200 import ShotBatch, configs
    vp = torch.full((ny, nz, nx), 3000., device="cuda")
    mu = 2000. * (vp / 1.8)**2
    b = ShotBatch()
    b.add(nx=nx, ny=ny, nz=nz, lenpml=W, dx=10., dt=0.0008, nt=NT,
          cpml=configs.cpml_profiles(20., 0.0008, 10., W, 3000., nx, ny, nz), lam=2000. * vp**2 - 2. * mu, mu=mu,
          rho=torch.full_like(vp, 2000.), wavelet=configs.ricker(25., 0.0008, NT), src=[[nx // 2, ny // 2, nz // 2]],
          mt=[[1., .5, -.5, .3, .2, .1]], rec=[[x, ny // 2, 2] for x in range(W, nx - W, 4)])
    return b


def _step_us(torch, b, gathers):
    def once():
        b.forward(save_borders=True, out=gathers)
        b.gradient(gathers, model=True, mt=True)

    once()
    times = []
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        once()
        once()
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1) / 2 / NT * 1e3)
    return float(np.min(times))


@pytest.mark.parametrize("grid", [(300, 44, 52, 8), (96, 96, 64, 10)], ids=str)
def test_unpaired_launches_choose_their_own_chunks(cuda, grid):
    from elastic_fm_vp_vs_rho_b200 import _lib
    b = _batch(cuda, *grid)
    b.set_option(_lib.EFM_OPT_PAIR_LAUNCH, 0)
    gathers = b.forward(save_borders=True)
    chosen = _step_us(cuda, b, gathers)
    by_hand = []
    for yc in (4, 5, 6):
        b.set_option(_lib.EFM_OPT_YCHUNK, yc)
        by_hand.append(_step_us(cuda, b, gathers))
    b.status()
    b.close()
    assert chosen <= 1.14 * min(by_hand)
