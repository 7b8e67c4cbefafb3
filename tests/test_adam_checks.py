"""Adam's single launch takes only what it can be handed: the kernel gets addresses and the
parameters' sizes, so every other form goes to the tensor operations, which raise or broadcast as
they always did."""
import ctypes

import pytest
import torch

from elastic_fm_vp_vs_rho_b200 import precond


class _OnDevice(torch.Tensor):
    """A CPU tensor that says it lives on a GPU (device 0 unless `index` says otherwise)."""
    index = 0
    is_cuda = property(lambda self: True)
    device = property(lambda self: torch.device("cuda", self.index))


def _fake(t, index=0):
    t = t.as_subclass(_OnDevice)
    t.index = index
    return t


class _Library:
    """Records the calls of efm_adam_step."""

    def __init__(self):
        self.sizes = []

    def efm_adam_step(self, n, p, g, m, v, sizes, *rest):
        self.sizes.append(list(sizes))
        return 0


@pytest.fixture
def step(monkeypatch):
    lib = _Library()
    monkeypatch.setattr(precond._lib, "load", lambda: lib)
    monkeypatch.setattr(precond, "stream_ptr", lambda *a: ctypes.c_void_p(0))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 0)

    def run(params, grads, moments=None):
        net = precond.PreconditionerNet(widths=(16, 16), device="cpu")
        net.parameters = lambda: params
        net.prep = lambda: None
        net._adam = moments or [tuple(_fake(torch.zeros(p.shape)) for _ in range(2)) for p in params]
        net.adam_step([(grads[i], grads[i + 1]) for i in range(0, len(grads), 2)], lr=0.1)
        return lib.sizes

    return run


def _tensors(*shapes):
    return [_fake(torch.ones(s)) for s in shapes]


def test_matching_tensors_take_one_launch(step):
    assert step(_tensors((3, 4), (4,)), _tensors((3, 4), (4,))) == [[12, 4]]


@pytest.mark.parametrize("shape", [(3, 3), (11,), (4, 3), (12,)], ids=str)
def test_gradients_of_another_shape_raise(step, shape):
    """Fewer elements (the kernel would read past them), or as many in another order."""
    with pytest.raises(RuntimeError):
        step(_tensors((3, 4), (4,)), _tensors(shape, (4,)))


def test_moments_of_another_shape_raise(step):
    m = [(_fake(torch.zeros(3, 3)), _fake(torch.zeros(3, 4))), (_fake(torch.zeros(4)), _fake(torch.zeros(4)))]
    with pytest.raises(RuntimeError):
        step(_tensors((3, 4), (4,)), _tensors((3, 4), (4,)), m)


def test_broadcast_gradients_and_short_lists_stay_with_tensor_operations(step):
    p = _tensors((3, 4), (4,))
    assert step(p, _tensors((1, 4), (4,))) == []
    assert float((p[0] - 0.9).abs().max()) < 1e-6  # one step of lr against a gradient of ones
    p = _tensors((3, 4), (4,), (5,), (2,))
    assert step(p, _tensors((3, 4), (4,))) == []
    assert float(p[2].min()) == 1.0 and float(p[0].max()) < 1.0


@pytest.mark.parametrize("which", [0, 1, 2])
def test_tensors_of_another_device_stay_with_tensor_operations(step, which):
    p, g = _tensors((3, 4), (4,)), _tensors((3, 4), (4,))
    m = [tuple(_fake(torch.zeros(q.shape)) for _ in range(2)) for q in p]
    (p[1] if which == 0 else g[1] if which == 1 else m[1][1]).index = 1
    assert step(p, g, m) == []


@pytest.mark.gpu
def test_gradient_of_another_shape_raises_on_the_gpu(cuda):
    net = precond.PreconditionerNet(widths=(16, 32, 16))
    grads = [(cuda.zeros_like(L.w), cuda.zeros_like(L.b)) for L in net.layers]
    w = grads[0][0]
    with pytest.raises(RuntimeError):
        net.adam_step([(w.reshape(27, 16, 32), grads[0][1])] + grads[1:])


@pytest.mark.gpu
def test_moments_and_updates_to_their_own_scale(cuda):
    """Against float64, each to the scale of its largest entry: the moments are three or four float32
    roundings per step (3 steps: 12 x 2^-24 = 7e-7); the parameters' changes a dozen (2e-6) and the
    rounding of the parameters themselves (3 x 2^-24 of the largest)."""
    gen = cuda.Generator().manual_seed(5)
    net = precond.PreconditionerNet(widths=(16, 32, 16))
    start = [p.cpu().double() for p in net.parameters()]
    ref = [p.clone() for p in start]
    mom = [(p * 0, p * 0) for p in ref]
    for step in range(1, 4):
        gs = [0.1 * cuda.randn(p.shape, generator=gen) for p in ref]
        net.adam_step([(gs[i].cuda(), gs[i + 1].cuda()) for i in range(0, len(gs), 2)], lr=1e-2)
        for p, g, (m, v) in zip(ref, gs, mom):
            g = g.double()
            m.mul_(0.9).add_(g, alpha=0.1)
            v.mul_(0.999).addcmul_(g, g, value=0.001)
            p.sub_(1e-2 * (m / (1 - 0.9**step)) / ((v / (1 - 0.999**step)).sqrt() + 1e-8))
    for p, r, s, (m, v), (m64, v64) in zip(net.parameters(), ref, start, net._adam, mom):
        for a, b in ((m, m64), (v, v64)):
            assert float((a.cpu().double() - b).abs().max()) <= 1e-6 * float(b.abs().max())
        change = float((r - s).abs().max())
        assert float((p.cpu().double() - r).abs().max()) <= 2e-6 * change + 3 * 2.0**-24 * float(r.abs().max())


@pytest.mark.gpu
def test_one_launch_rounds_as_the_tensor_operations_do(cuda):
    """Bit for bit what the elementwise operations give, moments and parameters, over five steps."""
    gen = cuda.Generator(device="cuda").manual_seed(7)
    net = precond.PreconditionerNet(widths=(16, 32, 16))
    ref = [p.clone() for p in net.parameters()]
    mom = [(cuda.zeros_like(p), cuda.zeros_like(p)) for p in ref]
    lr, b1, b2, eps = 1e-2, 0.9, 0.999, 1e-8
    for step in range(1, 6):
        gs = [0.1 * cuda.randn(p.shape, device="cuda", generator=gen) for p in ref]
        net.adam_step([(gs[i], gs[i + 1]) for i in range(0, len(gs), 2)], lr=lr)
        for p, g, (m, v) in zip(ref, gs, mom):
            m.mul_(b1).add_(g, alpha=1.0 - b1)
            v.mul_(b2).addcmul_(g, g, value=1.0 - b2)
            p.addcdiv_(m / (1.0 - b1**step), (v / (1.0 - b2**step)).sqrt_().add_(eps), value=-lr)
    for p, r, (m, v), (m2, v2) in zip(net.parameters(), ref, net._adam, mom):
        assert cuda.equal(m, m2) and cuda.equal(v, v2) and cuda.equal(p, r)
