"""The kernels of a model update at the sizes where their tiles, groups and strips can go wrong,
against float64 (the direction) and the oracle (smoothing and mask)."""
import numpy as np
import pytest

import efm_oracle as O

pytestmark = pytest.mark.gpu


def _two_loop(sk, yk, g, L, it):
    used = it if it < L else L - 1
    q, sig, eps = g.copy(), [], []
    for k in range(used):
        d = float(yk[k + 1] @ sk[k + 1])
        sig.append(0.0 if d == 0 else 1.0 / d)
        eps.append(sig[k] * float(sk[k + 1] @ q))
        q -= eps[k] * yk[k + 1]
    d = float(yk[1] @ yk[1])
    q *= 0.0 if d == 0 else float(sk[1] @ yk[1]) / d
    for k in range(used, 0, -1):
        q += sk[k] * (eps[k - 1] - sig[k - 1] * float(yk[k] @ q))
    return q


@pytest.mark.parametrize("n", [1, 37, 4096, 100_001, 262_148])
@pytest.mark.parametrize("layers,it", [(2, 0), (2, 1), (3, 7), (5, 4), (6, 4), (6, 5), (10, 8), (10, 9), (14, 13),
                                       (28, 26), (90, 88)])
def test_lbfgs_direction_and_history(cuda, n, layers, it):
    """Groups of four vectors (full, partial, one to seven of them), one and several tiles per
    block, vector lengths on and off 16 bytes.  The direction is rounded to float32 once; its
    coefficients are float64 sums of exact products: 2e-7 of its largest entry, times ten for
    the recursion's own conditioning."""
    from elastic_fm_vp_vs_rho_b200 import L_BFGS, compute_sk_yk
    rng = np.random.default_rng(n + layers)
    diag = 0.5 + rng.random(n)
    sk = np.zeros((layers, n), np.float32)
    yk = np.zeros((layers, n), np.float32)
    for k in range(min(layers - 1, it + 1)):
        sk[k] = rng.standard_normal(n)
        yk[k] = diag * sk[k] + 0.1 * rng.standard_normal(n)
    m, g = (rng.standard_normal(n).astype(np.float32) for _ in range(2))
    ds, dy, dm, dg = (cuda.as_tensor(a).cuda() for a in (sk, yk, m, g))
    compute_sk_yk(ds, dy, dm, dg, layers, it)
    if it == 0:
        ws, wy = np.concatenate([m[None], sk[1:]]), np.concatenate([g[None], yk[1:]])
    else:
        ws = np.concatenate([m[None], (m - sk[0])[None], sk[1:max(layers - 2, 1)], sk[layers - 1:]])[-layers:]
        wy = np.concatenate([g[None], (g - yk[0])[None], yk[1:max(layers - 2, 1)], yk[layers - 1:]])[-layers:]
        if layers == 2:
            ws, wy = np.stack([m, sk[1]]), np.stack([g, yk[1]])
    np.testing.assert_array_equal(ds.cpu().numpy(), ws)
    np.testing.assert_array_equal(dy.cpu().numpy(), wy)
    r = L_BFGS(ds, dy, dg, layers, it).cpu().numpy()
    ref = _two_loop(ws.astype(np.float64), wy.astype(np.float64), g.astype(np.float64), layers, it)
    assert np.abs(r - ref).max() <= 2e-6 * max(np.abs(ref).max(), 1e-30)


@pytest.mark.parametrize("shape,width", [((30, 26, 34), 3), ((9, 8, 7), 0), ((17, 41, 68), 2), ((6, 6, 12_100), 0),
                                         ((64, 33, 128), 8)])
@pytest.mark.parametrize("sigma", [0.0, 0.1, 1.0, 2.7, 4.0])
def test_smooth_mask_edges(cuda, shape, width, sigma):
    """Strips with remainders, rows on and off 16 bytes and too long for shared memory, radii from
    none to 16 (also past the volume's size).  Three passes of at most 33 float32 products: 6e-6."""
    from elastic_fm_vp_vs_rho_b200 import smooth_mask
    a = np.random.default_rng(3).standard_normal(shape).astype(np.float32)
    ref = O.postprocess_gradient(a, width=width, sigma=sigma, top=2)
    t = cuda.as_tensor(a).cuda()
    smooth_mask(t, sigma=sigma, lenpml=width, top=2)
    assert np.abs(t.cpu().numpy() - ref).max() <= 6e-6 * max(np.abs(ref).max(), 1e-30)


@pytest.mark.parametrize("count", [1, 8, 19])
def test_adam_step_matches_tensor_operations(cuda, count):
    """Tensors of unlike sizes, more of them than one launch takes; against the elementwise operations
    of the step in float64: a dozen float32 roundings, 1e-6 of the largest entry."""
    from elastic_fm_vp_vs_rho_b200.precond import PreconditionerNet
    rng = np.random.default_rng(count)
    net = PreconditionerNet(seed=0)
    ps = [rng.standard_normal(1 + 97 * k * k) for k in range(2 * ((count + 1) // 2))]
    net.parameters = lambda: par
    net.prep = lambda: None
    par = [cuda.as_tensor(p.astype(np.float32)).cuda() for p in ps]
    ref = [p.cpu().double() for p in par]
    mom = [(p * 0, p * 0) for p in ref]
    for step in range(1, 4):
        gs = [cuda.as_tensor(rng.standard_normal(p.numel()).astype(np.float32)).cuda() for p in par]
        net.adam_step(list(zip(gs[::2], gs[1::2])), lr=1e-2)
        for p, g, (m, v) in zip(ref, gs, mom):
            g = g.cpu().double()
            m.mul_(0.9).add_(g, alpha=0.1)
            v.mul_(0.999).addcmul_(g, g, value=0.001)
            p.sub_(1e-2 * (m / (1 - 0.9**step)) / ((v / (1 - 0.999**step)).sqrt() + 1e-8))
    for p, r, (m, v), (m64, v64) in zip(par, ref, net._adam, mom):
        for a, b in ((p, r), (m, m64), (v, v64)):
            assert float((a.cpu().double() - b).abs().max()) <= 1e-6 * max(1.0, float(b.abs().max()))
