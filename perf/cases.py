"""Performance cases: the work users of this package have it do, through its public entry points.

Each case is a dict of plain values; ``listed()`` gives the fixed ones and ``draw(rng)`` one more
of the same ranges.  Kinds:

* ``forward``  -- forward modelling of a batch of shots on one grid (observed data, trial misfits);
* ``gradient`` -- one evaluation of the inversion: forward with boundary strips, residual, imaging
  gradient for lambda / mu / rho and the moment tensor;
* ``uneven``   -- the same evaluation for a batch of different grids and record lengths;
* ``tensor``   -- moment-tensor inversion: forward, residual, moment-tensor gradient only;
* ``exact``    -- exact gradient through the torch.autograd bridge (Vp, Vs, rho, moment tensor);
* ``update``   -- what an inversion does with a gradient: chain rule, smoothing and masking, L-BFGS
  history and direction;
* ``conv``     -- one 3x3x3 convolution layer of the learned preconditioner, forward, data and
  weight gradient;
* ``train``    -- one training step of the learned preconditioner's network.

Record lengths are shorter than an inversion's (every step costs the same), grids, absorbing widths,
receiver and source counts are those of the package's workloads (``configs``, ``gradbench``,
``precond``) and of its tests.
"""
import math

import numpy as np
import torch

from elastic_fm_vp_vs_rho_b200 import ShotBatch, chain_rule, compute_sk_yk, configs, conv3d, smooth_mask
from elastic_fm_vp_vs_rho_b200 import L_BFGS
from elastic_fm_vp_vs_rho_b200.autograd import misfit
from elastic_fm_vp_vs_rho_b200.precond import PreconditionerNet, mse_grad


def listed():
    return [
        # plain forward workload: one shot on the smallest grid, 600 short steps (launch bound)
        dict(name="forward_64", kind="forward", nx=64, ny=64, nz=64, width=10, nt=600, shots=1, side=8),
        # observed data of several shots of the batched inversion in one batch
        dict(name="forward_200x4", kind="forward", nx=200, ny=200, nz=100, width=10, nt=200, shots=4, side=32),
        # one shot's gradient on the single-shot gradient grid
        dict(name="gradient_128", kind="gradient", nx=128, ny=128, nz=96, width=10, nt=300, shots=1, side=16),
        # the largest single-GPU shot (the headline grid)
        dict(name="gradient_256", kind="gradient", nx=256, ny=256, nz=128, width=10, nt=300, shots=1, side=48),
        # a grid whose rows are no multiple of a vector, two earthquakes
        dict(name="gradient_odd", kind="gradient", nx=121, ny=107, nz=83, width=10, nt=300, shots=2, side=11),
        # earthquakes on grids of their own with 1-4 sources each, one batch
        dict(name="uneven_6", kind="uneven", grids=4, count=6, nt=240),
        # moment-tensor inversion on the default regional grid (1 km cells, wide absorbing frame)
        dict(name="tensor_100", kind="tensor", nx=100, ny=100, nz=100, width=20, nt=300, shots=1, side=14),
        # exact gradients: the small inversion problem of the learned preconditioner ...
        dict(name="exact_48", kind="exact", nx=48, ny=48, nz=40, width=8, nt=320, shots=4, side=8),
        # ... and two shots on the single-shot gradient grid
        dict(name="exact_128", kind="exact", nx=128, ny=128, nz=96, width=10, nt=200, shots=2, side=16),
        # the update of one inversion iteration on the batched inversion's grid
        dict(name="update_200", kind="update", nx=200, ny=200, nz=100, width=10, layers=10, pairs=8),
        # the widest layer of the preconditioner on the single-shot grid
        dict(name="conv_32_64", kind="conv", nx=128, ny=128, nz=96, cin=32, cout=64),
        # a training step on the small inversion grid
        dict(name="train_48", kind="train", nx=48, ny=48, nz=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "gradient", "gradient", "gradient", "uneven", "tensor", "exact",
                       "exact", "update", "conv", "train"])
    if kind == "uneven":
        return dict(kind=kind, grids=rng.randint(10, 10 ** 6), count=rng.randint(2, 4), nt=rng.randint(160, 240))
    if kind == "conv":
        while True:
            cin, cout = rng.choice([16, 32, 64]), rng.choice([16, 32, 64])
            if (cin, cout) != (64, 64):
                break
        return dict(kind=kind, nx=_log(rng, 40, 200), ny=_log(rng, 40, 128), nz=_log(rng, 36, 96), cin=cin, cout=cout)
    if kind == "train":
        return dict(kind=kind, nx=_log(rng, 40, 128), ny=_log(rng, 40, 128), nz=_log(rng, 36, 96))
    if kind == "update":
        layers = rng.randint(5, 10)
        return dict(kind=kind, nx=_log(rng, 48, 256), ny=_log(rng, 48, 256), nz=_log(rng, 40, 128),
                    width=rng.choice([8, 10, 20]), layers=layers, pairs=rng.randint(1, layers + 2))
    width = rng.choice([8, 10, 10, 20])
    top = 128 if kind == "exact" else 256
    nx, ny, nz = _log(rng, 48, top), _log(rng, 48, top), _log(rng, 40, 96 if kind == "exact" else 128)
    if rng.random() < 0.5:
        nx = max(48, nx // 8 * 8)  # users mostly take round grid sizes
    nt = rng.randint(160, 240) if kind == "exact" else rng.randint(160, 320)
    # no more cell updates than the largest listed case of the kind
    most = (400_000_000 if kind == "exact" else 2_500_000_000) // (nx * ny * nz * nt)
    shots = 1 if kind == "tensor" else max(1, min(most, rng.choice([1, 1, 2, 4])))
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, width=width, nt=nt, shots=shots,
                side=rng.randint(6, max(6, min(32, min(nx, ny) - 2 * width))))


# ------------------------------------------------------------------------------------ inputs
def _model(rng, ny, nz, nx, dx, smooth=0.0):
    """Layered Vp 2000-4600 m/s with three Gaussian anomalies, Vs = Vp / 1.75, Gardner density: the
    layered models of ``configs``, built on the GPU.  float32 (ny, nz, nx) tensors."""
    z = torch.arange(nz, device="cuda", dtype=torch.float64)
    cuts = sorted(rng.integers(nz // 8, nz - nz // 8, 4))
    vels = np.sort(rng.uniform(2000.0, 4600.0, 5))
    prof = torch.full((nz,), float(vels[0]), device="cuda", dtype=torch.float64)
    for c, lo, hi in zip(cuts, vels[:-1], vels[1:]):
        step = torch.sigmoid((z - float(c)) / smooth) if smooth else (z >= float(c)).double()
        prof = prof + (float(hi) - float(lo)) * step
    vp = prof[None, :, None].expand(ny, nz, nx).clone()
    y = torch.arange(ny, device="cuda", dtype=torch.float64)
    x = torch.arange(nx, device="cuda", dtype=torch.float64)
    for _ in range(3):
        c = rng.uniform(0.3, 0.7, 3) * (ny, nz, nx)
        sg = 0.1 if rng.uniform() < 0.5 else -0.1
        w = 80.0 / dx
        g = (torch.exp(-((y - c[0]) / w) ** 2 / 2)[:, None, None] * torch.exp(-((z - c[1]) / w) ** 2 / 2)[None, :, None]
             * torch.exp(-((x - c[2]) / w) ** 2 / 2)[None, None, :])
        vp = vp * (1.0 + sg * g)
    rho = 310.0 * vp.pow(0.25)
    return vp.float().contiguous(), (vp / 1.75).float().contiguous(), rho.float().contiguous()


def _lame(vp, vs, rho):
    mu = (vs * vs * rho).contiguous()
    return (vp * vp * rho - 2.0 * mu).contiguous(), mu


def _instance(rng, nx, ny, nz, width, nt, side, dx=10.0, nsrc=1, model=None):
    """The keyword arguments of ShotBatch.add for one earthquake, and its seeded records."""
    vp, vs, rho = model if model is not None else _model(rng, ny, nz, nx, dx, smooth=15.0 if nz > 60 else 5.0)
    lam, mu = _lame(vp, vs, rho)
    dt = float(np.float32(0.4 * dx / 5100.0))
    fq = math.sqrt(2.0) / (max(50, nt // 4) * dt)  # the wavelet peaks after a quarter of the record
    cp = configs.cpml_profiles(fq, dt, dx, width, 5000.0, nx, ny, nz)
    rx, ry, rz = configs.surface_receivers(nx, ny, width, side, side)
    rec = np.stack([rx, ry, rz], axis=1)
    # sources below a station, as deep as the record lets their waves come back from
    near = rec[rng.integers(0, len(rec), nsrc)] + rng.integers(-5, 6, (nsrc, 3))
    top = min(nz - width - 4, 5 + nt // 20)
    src = np.stack([np.clip(near[:, 0], width + 3, nx - width - 4), np.clip(near[:, 1], width + 3, ny - width - 4),
                    rng.integers(4, top + 1, nsrc)], axis=1).astype(np.int32)
    mt = np.stack([configs.random_moment_tensor(rng) for _ in range(nsrc)])
    kw = dict(nx=nx, ny=ny, nz=nz, lenpml=width, dx=dx, dt=dt, nt=nt, cpml=cp, lam=lam, mu=mu, rho=rho,
              wavelet=torch.as_tensor(configs.ricker(fq, dt, nt)).cuda(), src=src, mt=mt, rec=rec)
    # observed records: a Ricker arrival per receiver at its distance's travel time, seeded sizes
    d = torch.as_tensor(np.linalg.norm((rec - src[0]) * dx, axis=1), device="cuda", dtype=torch.float64)
    t = torch.arange(nt, device="cuda", dtype=torch.float64)[:, None] * dt
    a = (math.pi * fq * (t - math.sqrt(2.0) / fq - d[None, :] / 3200.0)) ** 2
    amp = torch.as_tensor(rng.standard_normal((3, 1, len(rec))), device="cuda") * (2e-8 / (1.0 + d / dx))
    return kw, (amp * ((1 - 2 * a) * torch.exp(-a))[None]).float().reshape(-1)


def _uneven_instances(case, seed):
    """Grids between 64^3 and 160 x 160 x 96 fixed by the case, everything else by the seed."""
    shape, rng = np.random.default_rng(case["grids"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["count"]):
        nx, ny = (int(shape.integers(8, 21)) * 8 for _ in range(2))
        nz, side, nsrc = int(shape.integers(64, 97)), int(shape.integers(8, 17)), int(shape.integers(1, 5))
        nt = int(case["nt"] * shape.uniform(0.7, 1.0))
        out.append(_instance(rng, nx, ny, nz, 10, nt, side, dx=float(np.float32(shape.uniform(10.0, 20.0))),
                             nsrc=nsrc))
    return out


def _instances(case, seed):
    if case["kind"] == "uneven":
        return _uneven_instances(case, seed)
    rng = np.random.default_rng(seed)
    far = case["kind"] == "tensor"
    model = _model(rng, case["ny"], case["nz"], case["nx"], 10.0, smooth=15.0 if case["nz"] > 60 else 5.0)
    return [_instance(rng, case["nx"], case["ny"], case["nz"], case["width"], case["nt"], case["side"],
                      dx=1000.0 if far else 10.0, model=model)
            for _ in range(case["shots"])]


def _randn(gen, *shape, dtype=torch.float32):
    return torch.randn(shape, generator=gen, device="cuda").to(dtype)


def _update_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape, rng = (case["ny"], case["nz"], case["nx"]), np.random.default_rng(seed)
    model = _model(rng, *shape, 10.0, smooth=5.0)
    L = case["layers"]
    # curvature pairs of a positive operator with seeded noise, newest first; layer L-1 unwritten
    sk, yk = torch.zeros((L,) + shape, device="cuda"), torch.zeros((L,) + shape, device="cuda")
    diag = 0.5 + torch.rand(shape, generator=g, device="cuda")
    for k in range(1, min(L - 1, case["pairs"] + 1)):
        sk[k] = _randn(g, *shape)
        yk[k] = diag * sk[k] + 0.1 * _randn(g, *shape)
    sk[0], yk[0] = _randn(g, *shape), _randn(g, *shape)
    step = _randn(g, *shape)
    # two models an inversion moves between, and their gradients
    at = [(sk[0] + step, yk[0] + diag * step + 0.1 * _randn(g, *shape)), (sk[0].clone(), yk[0].clone())]
    grad = [_randn(g, *shape) for _ in range(3)]
    return dict(sk=sk, yk=yk, at=at, grad=grad, model=model, tmp=torch.empty(shape, device="cuda"))


def _conv_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    vol = (case["ny"], case["nz"], case["nx"])
    cin, cout = case["cin"], case["cout"]
    x = _randn(g, *vol, cin).clamp_min(0).to(torch.bfloat16)  # a ReLU layer's output
    dy = _randn(g, *vol, cout, dtype=torch.bfloat16)
    w = _randn(g, 27, cout, cin) * math.sqrt(2.0 / (27 * cin))
    return dict(x=x, dy=dy, w=w, b=0.1 * _randn(g, cout))


def _train_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    vol = (case["ny"], case["nz"], case["nx"])
    x = _randn(g, *vol, 16)
    x[..., 8:] = 0  # features fill eight of the sixteen channels
    return x.to(torch.bfloat16), _randn(g, *vol, 3)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "update":
        return dict(case=case, **_update_inputs(case, seed))
    if kind == "conv":
        s = _conv_inputs(case, seed)
        s["wb"], s["wt"] = conv3d.prep_weights(s["w"])
        return dict(case=case, ws=conv3d.WgradWorkspace(), **s)
    if kind == "train":
        x, t = _train_inputs(case, seed)
        return dict(case=case, x=x, t=t, net=PreconditionerNet(seed=seed % 997))
    batch, obs = ShotBatch(), []
    for kw, o in _instances(case, seed):
        batch.add(**kw)
        obs.append(o)
    s = dict(case=case, batch=batch, obs=torch.cat(obs))
    if kind == "exact":
        rng = np.random.default_rng(seed)
        s["model"] = [p.requires_grad_(True) for p in
                      _model(rng, case["ny"], case["nz"], case["nx"], 10.0, smooth=15.0 if case["nz"] > 60 else 5.0)]
        s["mt"] = torch.as_tensor(np.stack([sp["mt"] for sp in batch.specs]), device="cuda").requires_grad_(True)
    return s


# ------------------------------------------------------------------------------------- a pass
def run(s):
    kind = s["case"]["kind"]
    if kind == "update":
        sk, yk, tmp, case = s["sk"], s["yk"], s["tmp"], s["case"]
        g = [t.clone() for t in s["grad"]]
        chain_rule(*g, *s["model"])
        for t in g:
            smooth_mask(t, sigma=1.0, lenpml=case["width"], top=10, tmp=tmp)
        m, gk = s["at"][0]
        s["at"].reverse()  # the next iteration is at the other model: its step is not zero
        compute_sk_yk(sk, yk, m, gk, case["layers"], case["pairs"])
        return dict(grad=g, sk=sk, yk=yk, r=L_BFGS(sk, yk, gk, case["layers"], case["pairs"]))
    if kind == "conv":
        y, _ = conv3d.forward(s["x"], s["wb"], s["b"], relu=True)
        dx = conv3d.backward_data(s["dy"], s["wt"], s["case"]["cin"], relu_mask=s["x"])
        dw, db = conv3d.backward_weights(s["x"], s["dy"], s["ws"])
        return dict(y=y, dx=dx, dw=dw, db=db)
    if kind == "train":
        net = s["net"]
        out = net.forward(s["x"], keep=True)
        _, d = mse_grad(out, s["t"])
        grads = net.backward(d)
        net.adam_step(grads, lr=0.0)  # the step's work, the same weights for the next pass
        return dict(out=out, dw=[a for a, _ in grads], db=[b for _, b in grads])
    batch = s["batch"]
    if kind == "forward":
        return batch.forward()
    if kind == "exact":
        for p in (*s["model"], s["mt"]):
            p.grad = None
        misfit(*s["model"], s["mt"], batch, s["obs"]).backward()
        return [p.grad for p in s["model"]] + [s["mt"].grad]
    mod = batch.forward(save_borders=kind != "tensor")
    res, _ = batch.residual_misfit(mod, s["obs"])
    g, m = batch.gradient(res, model=kind != "tensor", mt=True)
    # moment tensors and their updates are float32 in an inversion, as in the autograd bridge
    return dict(mod=mod, res=res, mt=m.float(), **({} if g is None else {"grad": g}))


# --------------------------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "update":
        n, m = case["nx"] * case["ny"] * case["nz"], min(case["pairs"], case["layers"] - 1)
        # gradients and model in, gradients out, both histories in and out, new model and gradient in,
        # direction out
        return dict(bytes=4 * n * (3 + 3 + 3 + 4 * (case["layers"] - 1) + 2 + 1), flops=n * (60 + 12 * m))
    if kind == "conv":
        n, c = case["nx"] * case["ny"] * case["nz"], case["cin"] + case["cout"]
        return dict(bytes=2 * n * 2 * c, flops=6.0 * 27 * case["cin"] * case["cout"] * n)
    if kind == "train":
        n = case["nx"] * case["ny"] * case["nz"]
        pairs = 16 * 32 + 32 * 64 + 64 * 32 + 32 * 16
        return dict(bytes=n * (2 * 16 + 12 + 64 + 2 * 2 * (32 + 64 + 32)), flops=2.0 * 27 * n * (3 * pairs - 16 * 32))
    if kind == "uneven":
        shape, cells = np.random.default_rng(case["grids"]), 0
        for _ in range(case["count"]):
            nx, ny = (int(shape.integers(8, 21)) * 8 for _ in range(2))
            nz = int(shape.integers(64, 97))
            shape.integers(8, 17), shape.integers(1, 5)
            cells += nx * ny * nz * int(case["nt"] * shape.uniform(0.7, 1.0))
            shape.uniform(10.0, 20.0)
    else:
        cells = case["nx"] * case["ny"] * case["nz"] * case["shots"] * case["nt"]
    # per cell and step: 9 fields in and out and the 3 model volumes (84 bytes); the imaging gradient
    # steps two such states and adds into 3 volumes (192); the exact one reads the stored forward
    # states (36 bytes, written by the forward) and its own state, model and gradients (108)
    b, f = {"forward": (84, 110), "gradient": (84 + 192, 400), "uneven": (84 + 192, 400), "tensor": (168, 220),
            "exact": (84 + 36 + 36 + 108, 420)}[kind]
    return dict(bytes=float(b) * cells, flops=float(f) * cells)


# ------------------------------------------------------------------------ the same in 64 bits
def _sh(a, y=0, z=0, x=0):
    """The interior (two cells off every face) of a, shifted."""
    ny, nz, nx = a.shape
    return a[2 + y:ny - 2 + y, 2 + z:nz - 2 + z, 2 + x:nx - 2 + x]


def _pad(a):
    return torch.nn.functional.pad(a, (2, 2, 2, 2, 2, 2))


class _Scheme:
    """The staggered velocity-stress scheme in float64: state (v, t, p) of three velocities, six
    stresses (xx yy zz xy xz yz) and 18 interior memory variables."""

    def __init__(self, kw, lam=None, mu=None, rho=None):
        f = lambda a: torch.as_tensor(np.asarray(a, np.float32) if not torch.is_tensor(a) else a).double().cuda()  # noqa: E731
        self.shape = (kw["ny"], kw["nz"], kw["nx"])
        self.k = float(np.float32(kw["dt"]) / np.float32(kw["dx"]))
        self.dt, self.dx = float(np.float32(kw["dt"])), float(np.float32(kw["dx"]))
        cp = {n: f(v)[2:-2] for n, v in kw["cpml"].items()}
        ax = {"x": (1, 1, -1), "y": (-1, 1, 1), "z": (1, -1, 1)}
        self.a = {d: cp["a" + d].view(s) for d, s in ax.items()}
        self.b = {d: cp["b" + d].view(s) for d, s in ax.items()}
        self.w, self.src = f(kw["wavelet"]), kw["src"]
        self.mt = f(kw["mt"]).reshape(-1, 6)
        self.rec = tuple(torch.as_tensor(kw["rec"][:, c]).long().cuda() for c in (1, 2, 0))
        self.model(*(f(kw[n]) if v is None else v for n, v in (("lam", lam), ("mu", mu), ("rho", rho))))

    def model(self, lam, mu, rho):
        r = 1.0 / mu
        c = _sh(r)
        self.lam, self.mu0 = _sh(lam), _sh(mu)
        self.mxy = 4.0 / (c + _sh(r, x=1) + _sh(r, y=1) + _sh(r, y=1, x=1))
        self.mxz = 4.0 / (c + _sh(r, x=1) + _sh(r, z=1) + _sh(r, z=1, x=1))
        self.myz = 4.0 / (c + _sh(r, y=1) + _sh(r, z=1) + _sh(r, y=1, z=1))
        self.B = [2.0 / (_sh(rho) + _sh(rho, **{d: 1})) for d in "xyz"]

    def zero(self):
        z = lambda: torch.zeros(self.shape, dtype=torch.float64, device="cuda")  # noqa: E731
        q = tuple(n - 4 for n in self.shape)
        return [z() for _ in range(3)], [z() for _ in range(6)], [torch.zeros(q, dtype=torch.float64, device="cuda")
                                                                 for _ in range(18)]

    def _damp(self, p, i, d, ds, out):
        for j, q in enumerate(ds):
            out[i + j] = self.b[d] * p[i + j] + self.a[d] * q
        return [q + out[i + j] for j, q in enumerate(ds)]

    def stress(self, v, t, p, sign=1.0, damp=True):
        vx, vy, vz = v
        dxs = [_sh(vx) - _sh(vx, x=-1), _sh(vy, x=1) - _sh(vy), _sh(vz, x=1) - _sh(vz)]
        dys = [_sh(vy) - _sh(vy, y=-1), _sh(vx, y=1) - _sh(vx), _sh(vz, y=1) - _sh(vz)]
        dzs = [_sh(vz) - _sh(vz, z=-1), _sh(vx, z=1) - _sh(vx), _sh(vy, z=1) - _sh(vy)]
        p = list(p)
        if damp:
            dxs, dys, dzs = (self._damp(p, i, d, s, p) for i, d, s in ((0, "x", dxs), (3, "y", dys), (6, "z", dzs)))
        ex, ey, ez = dxs[0], dys[0], dzs[0]
        k, tr = sign * self.k, ex + ey + ez
        inc = [k * (self.lam * tr + 2.0 * self.mu0 * e) for e in (ex, ey, ez)]
        inc += [k * self.mxy * (dys[1] + dxs[1]), k * self.mxz * (dzs[1] + dxs[2]), k * self.myz * (dzs[2] + dys[2])]
        return inc, p

    def velocity(self, t, p, sign=1.0, damp=True):
        txx, tyy, tzz, txy, txz, tyz = t
        dxs = [_sh(txx, x=1) - _sh(txx), _sh(txy) - _sh(txy, x=-1), _sh(txz) - _sh(txz, x=-1)]
        dys = [_sh(tyy, y=1) - _sh(tyy), _sh(txy) - _sh(txy, y=-1), _sh(tyz) - _sh(tyz, y=-1)]
        dzs = [_sh(tzz, z=1) - _sh(tzz), _sh(txz) - _sh(txz, z=-1), _sh(tyz) - _sh(tyz, z=-1)]
        p = list(p)
        if damp:
            dxs, dys, dzs = (self._damp(p, i, d, s, p) for i, d, s in ((9, "x", dxs), (12, "y", dys), (15, "z", dzs)))
        k = sign * self.k
        return [k * self.B[0] * (dxs[0] + dys[1] + dzs[1]), k * self.B[1] * (dxs[1] + dys[0] + dzs[2]),
                k * self.B[2] * (dxs[2] + dys[2] + dzs[0])], p

    def source(self, t, w, sign=1.0):
        for (x, y, z), m in zip(self.src, self.mt):
            for c in range(6):
                t[c][y, z, x] += sign * m[c] * w

    def step(self, v, t, p, it=None):
        """In place; with `it`, the source of that step."""
        inc, p = self.stress(v, t, p)
        for a, i in zip(t, inc):
            _sh(a).add_(i)
        if it is not None:
            self.source(t, self.w[it])
        inc, p = self.velocity(t, p)
        for a, i in zip(v, inc):
            _sh(a).add_(i)
        return v, t, p

    def pure_step(self, v, t, p, mt, w):
        """The step as a function of its arguments (for autograd)."""
        inc, p = self.stress(v, t, p)
        t = [a + _pad(i) for a, i in zip(t, inc)]
        hit = torch.zeros(self.shape, dtype=torch.float64, device="cuda")
        for n, (x, y, z) in enumerate(self.src):
            one = hit.clone()
            one[y, z, x] = w
            t = [a + one * mt[n, c] for c, a in enumerate(t)]
        inc, p = self.velocity(t, p)
        return [a + _pad(i) for a, i in zip(v, inc)], t, p


def _strips(kw):
    """Masks of the box inside the absorbing frame and of its two outer layers."""
    ny, nz, nx, w = kw["ny"], kw["nz"], kw["nx"], kw["lenpml"]
    box = torch.zeros((ny, nz, nx), dtype=torch.bool, device="cuda")
    box[w:ny - w, 2:nz - w, w:nx - w] = True
    inner = torch.zeros_like(box)
    inner[w + 2:ny - w - 2, 4:nz - w - 2, w + 2:nx - w - 2] = True
    return box, box & ~inner


def _imaging(S, kw, res, tail, strips, model):
    """Adjoint, reverse-time rebuild and zero-lag imaging of one instance from the forward's last
    state and its stored strips; res (3, nt, nrec) float64."""
    nt, w = kw["nt"], kw["lenpml"]
    ny, nz, nx = S.shape
    v, t, _ = tail
    bv, bt, bp = S.zero()
    grad = torch.zeros((3, ny, nz, nx), dtype=torch.float64, device="cuda")
    gmt = torch.zeros((4, 6), dtype=torch.float64, device="cuda")
    if model:
        box, strip = _strips(kw)
        keep = box.clone()
        keep[:, :2], keep[:, -2:], keep[:2], keep[-2:], keep[..., :2], keep[..., -2:] = (False,) * 6
        hold = torch.zeros_like(box)
        hold[w:ny - w, 2:nz - w, w:nx - w] = True
        hold_i = _sh(hold).double()
    for it in range(nt - 1 if model else nt):
        inc, bp = S.stress(bv, bt, bp)
        for a, i in zip(bt, inc):
            _sh(a).add_(i)
        for n, (x, y, z) in enumerate(S.src):  # strain of the adjoint stress at the source
            q = torch.stack([a[y, z, x] for a in bt])
            l, m = S.lam[y - 2, z - 2, x - 2], S.mu0[y - 2, z - 2, x - 2]
            f = 1.0 / (2.0 * m * (3.0 * l + 2.0 * m))
            e = torch.cat([f * (2.0 * (l + m) * q[:3] - l * (q[:3].sum() - q[:3])),
                           torch.stack([q[3 + j] / a[y - 2, z - 2, x - 2] for j, a in enumerate((S.mxy, S.mxz, S.myz))])])
            gmt[n] += S.w[nt - 1 - it] * e
        inc, bp = S.velocity(bt, bp)
        for a, i in zip(bv, inc):
            _sh(a).add_(i)
        for c in range(3):
            bv[c].index_put_(S.rec, res[c, nt - 1 - it], accumulate=True)
        if not model:
            continue
        old = [a.clone() for a in v]
        inc, _ = S.velocity(t, bp, -1.0, damp=False)
        for c in range(3):
            new = torch.where(keep, old[c], 0.0)
            _sh(new).add_(inc[c] * _sh(keep).double())
            new[strip] = strips[nt - 2 - it][c]
            v[c] = new
        _image(S, old, v, bv, bt, grad)
        inc, _ = S.stress(v, t, bp, -1.0, damp=False)
        for a, i in zip(t, inc):
            _sh(a).add_(i * hold_i)
        S.source(t, S.w[nt - 1 - it], -1.0)
    return grad, gmt


def _image(S, p, n, bv, bt, g):
    px, py, pz = p
    _sh(g[2]).sub_(sum(_sh(b) * (_sh(a) - _sh(c)) / S.dt for a, c, b in zip(p, n, bv)))
    e = [_sh(px) - _sh(px, x=-1), _sh(py) - _sh(py, y=-1), _sh(pz) - _sh(pz, z=-1)]
    div = (0.5 / S.dx) * (_sh(px) - _sh(px, x=-2) + _sh(py) - _sh(py, y=-2) + _sh(pz) - _sh(pz, z=-2))
    xx, yy, zz, xy, xz, yz = (_sh(a) for a in bt)
    tr, l, m = xx + yy + zz, S.lam, S.mu0
    _sh(g[0]).add_(tr * div / (3.0 * l + 2.0 * m))
    f = 1.0 / (m * (3.0 * l + 2.0 * m))
    gm = sum(f * (2.0 * (l + m) * a - l * (tr - a)) * d for a, d in zip((xx, yy, zz), e))
    gm += xy / S.mxy * (_sh(py, x=1) - _sh(py) + _sh(px, y=1) - _sh(px))
    gm += xz / S.mxz * (_sh(px, z=1) - _sh(px) + _sh(pz, x=1) - _sh(pz))
    gm += yz / S.myz * (_sh(pz, y=1) - _sh(pz) + _sh(py, z=1) - _sh(py))
    _sh(g[1]).add_(gm)


def _exact_shots(case, seed):
    kind = case["kind"]
    mods, ress, mts, grads = [], [], [], []
    for kw, obs in _instances(case, seed):
        S = _Scheme(kw)
        v, t, p = S.zero()
        mod = torch.zeros((3, kw["nt"], len(kw["rec"])), dtype=torch.float64, device="cuda")
        strip = _strips(kw)[1] if kind in ("gradient", "uneven") else None
        strips = []
        for it in range(kw["nt"]):
            v, t, p = S.step(v, t, p, it)
            for c in range(3):
                mod[c, it] = v[c][S.rec]
            if strip is not None:
                strips.append([a[strip] for a in v])
        mods.append(mod.reshape(-1))
        if kind == "forward":
            continue
        res = mod - obs.double().view_as(mod)
        g, m = _imaging(S, kw, res, (v, t, p), strips, kind != "tensor")
        ress.append(res.reshape(-1))
        grads.append(g.reshape(-1))
        mts.append(m)
    if kind == "forward":
        return torch.cat(mods)
    out = dict(mod=torch.cat(mods), res=torch.cat(ress), mt=torch.stack(mts))
    return out if kind == "tensor" else dict(out, grad=torch.cat(grads))


def _exact_gradient(case, seed):
    rng = np.random.default_rng(seed)
    leaves = [p.double().requires_grad_(True) for p in
              _model(rng, case["ny"], case["nz"], case["nx"], 10.0, smooth=15.0 if case["nz"] > 60 else 5.0)]
    total, gm = [torch.zeros_like(p) for p in leaves], []
    every = max(1, int(math.sqrt(case["nt"])))
    for kw, obs in _instances(case, seed):
        S = _Scheme(kw)
        mt = S.mt.clone().requires_grad_(True)
        obs = obs.double().view(3, kw["nt"], -1)
        mu = leaves[1] ** 2 * leaves[2]
        lam = leaves[0] ** 2 * leaves[2] - 2.0 * mu
        prm = [q.detach().requires_grad_(True) for q in (lam, mu, leaves[2])]
        S.model(*(q.detach() for q in prm))
        saved, state = [], S.zero()
        with torch.no_grad():
            for it in range(kw["nt"]):
                if it % every == 0:
                    saved.append([[a.clone() for a in part] for part in state])
                state = S.pure_step(*state, mt, S.w[it])
        acc = [torch.zeros_like(q) for q in prm] + [torch.zeros_like(mt)]
        bar = [torch.zeros_like(a) for part in state for a in part]
        for first in range((kw["nt"] - 1) // every * every, -1, -every):
            states = [saved[first // every]]
            with torch.no_grad():
                S.model(*(q.detach() for q in prm))
                for it in range(first, min(kw["nt"], first + every) - 1):
                    states.append(S.pure_step(*states[-1], mt, S.w[it]))
            for it in range(min(kw["nt"], first + every) - 1, first - 1, -1):
                ins = [a.detach().requires_grad_(True) for part in states.pop() for a in part]
                S.model(*prm)
                new = S.pure_step(ins[:3], ins[3:9], ins[9:], mt, S.w[it])
                outs = [a for part in new for a in part]
                for c in range(3):
                    bar[c].index_put_(S.rec, outs[c].detach()[S.rec] - obs[c, it], accumulate=True)
                got = torch.autograd.grad(outs, ins + prm + [mt], bar)
                bar = [a.clone() for a in got[:27]]
                for a, q in zip(acc, got[27:]):
                    a.add_(q)
        for a, q in zip(total, torch.autograd.grad((lam, mu), leaves, acc[:2])):
            a.add_(q)
        total[2].add_(acc[2])
        gm.append(acc[3])
    return total + [torch.stack(gm)]


def _gauss(a, axis):
    w = np.exp(-0.5 * np.arange(-4, 5) ** 2.0)
    w /= w.sum()
    n = a.shape[axis]
    i = np.arange(-4, n + 4)
    i = np.where(i < 0, -i - 1, np.where(i >= n, 2 * n - i - 1, i))
    b = a.index_select(axis, torch.as_tensor(i, device=a.device))
    return sum(float(c) * b.narrow(axis, j, n) for j, c in enumerate(w))


def _exact_update(case, seed):
    s = _update_inputs(case, seed)
    (vp, vs, rho), (l, m, r) = ([a.double() for a in q] for q in (s["model"], s["grad"]))
    g = [2 * rho * vp * l, 2 * rho * vs * (m - 2 * l), r + (vp * vp - 2 * vs * vs) * l + vs * vs * m]
    w = case["width"] + 2
    for a in range(3):
        for axis in range(3):
            g[a] = _gauss(g[a], axis)
        mask = torch.zeros_like(g[a])
        mask[w:-w, 10:-w, w:-w] = 1
        g[a] = g[a] * mask
    L, it = case["layers"], case["pairs"]
    sk, yk = s["sk"].double(), s["yk"].double()
    mk, gk = (a.double() for a in s["at"][0])
    sk = torch.cat([mk[None], (mk - sk[0])[None], sk[1:L - 2], sk[L - 1:]])
    yk = torch.cat([gk[None], (gk - yk[0])[None], yk[1:L - 2], yk[L - 1:]])
    used = it if it < L else L - 1
    dot = lambda a, b: float((a * b).sum())  # noqa: E731
    q, sig, eps = gk.clone(), [], []
    for k in range(used):
        d = dot(yk[k + 1], sk[k + 1])
        sig.append(0.0 if d == 0 else 1.0 / d)
        eps.append(sig[k] * dot(sk[k + 1], q))
        q -= eps[k] * yk[k + 1]
    d = dot(yk[1], yk[1])
    q *= 0.0 if d == 0 else dot(sk[1], yk[1]) / d
    for k in range(used, 0, -1):
        q += sk[k] * (eps[k - 1] - sig[k - 1] * dot(yk[k], q))
    return dict(grad=g, sk=sk, yk=yk, r=q)


def _taps(a, flip=False):
    """Per kernel tap the (voxels, channels) matrix of the zero-padded volume it reads."""
    ny, nz, nx, c = a.shape
    p = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1, 1, 1))
    for t in range(27):
        d, h, w = ((26 - t) if flip else t) // 9, ((26 - t) if flip else t) // 3 % 3, ((26 - t) if flip else t) % 3
        yield t, p[d:d + ny, h:h + nz, w:w + nx].reshape(-1, c)


def _conv64(x, w, b=None):
    y = torch.zeros((x[..., 0].numel(), w.shape[1]), dtype=torch.float64, device="cuda")
    for t, a in _taps(x):
        y.addmm_(a, w[t].T)
    return (y if b is None else y + b).view(*x.shape[:3], -1)


def _conv64_back(x, dy, w):
    dx = torch.zeros((x[..., 0].numel(), w.shape[2]), dtype=torch.float64, device="cuda")
    for t, a in _taps(dy, flip=True):
        dx.addmm_(a, w[t])
    flat = dy.reshape(-1, dy.shape[-1])
    dw = torch.stack([flat.T @ a for _, a in _taps(x)])
    return dx.view_as(x), dw, flat.sum(0)


def exact(case, seed):
    kind = case["kind"]
    if kind == "update":
        return _exact_update(case, seed)
    if kind == "conv":
        s = {k: v.double() for k, v in _conv_inputs(case, seed).items()}
        w = s["w"].to(torch.bfloat16).double()  # the layer's weights are bfloat16
        dx, dw, db = _conv64_back(s["x"], s["dy"], w)
        return dict(y=_conv64(s["x"], w, s["b"]).clamp_min(0), dx=dx * (s["x"] > 0), dw=dw, db=db)
    if kind == "train":
        x, t = (a.double() for a in _train_inputs(case, seed))
        net, acts = PreconditionerNet(seed=seed % 997), [x]
        ws = [(layer.w.to(torch.bfloat16).double(), layer.b.double()) for layer in net.layers]
        for i, (w, b) in enumerate(ws):
            y = _conv64(acts[-1], w, b)
            acts.append(y.clamp_min(0) if i < len(ws) - 1 else y)
        g = torch.zeros_like(acts[-1])
        g[..., :3] = (acts[-1][..., :3] - t) * (2.0 / t.numel())
        dws, dbs = [], []
        for i in reversed(range(len(ws))):
            dx, dw, db = _conv64_back(acts[i], g, ws[i][0])
            dws.insert(0, dw)
            dbs.insert(0, db)
            g = dx * (acts[i] > 0)
        return dict(out=acts[-1], dw=dws, db=dbs)
    return _exact_gradient(case, seed) if kind == "exact" else _exact_shots(case, seed)
