"""L-BFGS directions of long histories: the recursion on inner products and the one vector by vector.

The direction takes the vectors' recursion where the products would cost more: many pairs of large
vectors, and more than 1024 pairs of any, so that the scratch of the products stays bounded."""
import pytest

pytestmark = pytest.mark.gpu


def _history(torch, layers, n):
    gen = torch.Generator(device="cuda").manual_seed(layers)
    diag = 0.5 + torch.rand(n, device="cuda", generator=gen)
    s = torch.randn((layers, n), device="cuda", generator=gen)
    y = diag * s
    for row in y:
        row += 0.1 * torch.randn(n, device="cuda", generator=gen)
    return s, y, torch.randn(n, device="cuda", generator=gen)


def _two_loop(torch, s, y, g, used):
    q, sig, eps = g.double(), [], []
    for k in range(1, used + 1):
        sig.append(1.0 / float(y[k].double() @ s[k].double()))
        eps.append(sig[-1] * float(s[k].double() @ q))
        q -= eps[-1] * y[k].double()
    q *= float(s[1].double() @ y[1].double()) / float(y[1].double() @ y[1].double())
    for k in range(used, 0, -1):
        q += s[k].double() * (eps[k - 1] - sig[k - 1] * float(y[k].double() @ q))
    return q


@pytest.mark.parametrize("layers,n", [(66, 2_000_000), (98, 2_500_000), (98, 2_500_001), (130, 4_000), (1025, 3_000),
                                      (1026, 3_000), (1026, 3_001)])
def test_direction_of_a_long_history(cuda, layers, n):
    """Both sides of the rules.  Vector by vector the direction is rounded to float32 after each of
    its 2 (layers - 1) steps: 2^-24 of its largest entry each, added up, times ten for the
    recursion's own conditioning (the products round once)."""
    from elastic_fm_vp_vs_rho_b200 import L_BFGS
    s, y, g = _history(cuda, layers, n)
    ref = _two_loop(cuda, s, y, g, layers - 1)
    keep = g.clone()
    r = L_BFGS(s, y, g, layers, layers - 1)
    assert cuda.equal(g, keep)
    bound = 10 * 2 * (layers - 1) * 2.0**-24
    assert float((r.double() - ref).abs().max()) <= bound * float(ref.abs().max())


def test_scratch_of_thousands_of_layers_stays_bounded(cuda):
    """4000 layers: the products of all pairs would take 1.3 GB of the device, kept for good."""
    from elastic_fm_vp_vs_rho_b200 import L_BFGS
    s, y, g = _history(cuda, 4000, 16)
    L_BFGS(s[:3], y[:3], g, 3, 2)
    cuda.cuda.synchronize()
    free = cuda.cuda.mem_get_info()[0]
    r = L_BFGS(s, y, g, 4000, 3999)
    cuda.cuda.synchronize()
    assert free - cuda.cuda.mem_get_info()[0] <= 128 << 20
    assert r.shape == g.shape
