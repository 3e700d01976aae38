"""The work that users of this library have it do, as measurable cases.

Every case is one pass through the public entry points (fwi3d_b200.lib), with
inputs made from a seed:

  model     forward modeling of shots, seismograms to the host or to a device
            buffer (the modeling workflow);
  misfit    one misfit evaluation of an inversion: new velocity, modeling of a
            batch of shots behind Cerjan boundaries, FP64 residual (what the
            line search repeats for every trial model);
  rtm       migration of a batch of shots: forward, fused back-propagation,
            the raw image and illumination;
  gradient  one FWI gradient of a batch of shots: new velocity, forward, fused
            back-propagation with the gradient condition (d2/dy2 kept, source
            removed), the raw gradient and illumination;
  residual  the FP64 misfit of recorded against modelled data;
  post      the image from accumulators (after a sum over GPUs);
  cnn_forward, cnn_train
            the learned preconditioner on a model's volume.

Fields of a propagation case: nz, nx, ny (model cells), nb (pad cells), dh [m],
nt samples of dt, fmax [Hz], batch (shots per launch), shots (in the call),
rec (receiver spacing in cells), boundary, pad ("shot": the library's random
pad per shot, rebuilt in the pass as migrations and inversions have it;
"given": a padded velocity that the caller made), host (data and results in
host memory).  The sizes are those of fwi3d_b200/synth.py and of the tests,
with shorter time axes for the large grids: a time step costs the same early
and late.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fwi3d_b200 import lib

W = (2.847222222222, 1.6, -0.2, 0.025396825396, -0.001785714285)  # centre (negative), then taps 1..4


def _prop(name, kind, nz, nx, ny, nb, nt, batch, shots, rec, *, dh=10.0, dt=1e-3, fmax=30.0, pad="given",
          host=False):
    return dict(name=name, kind=kind, nz=nz, nx=nx, ny=ny, nb=nb, nt=nt, batch=batch, shots=shots, rec=rec, dh=dh,
                dt=dt, fmax=fmax, pad=pad, host=host)


def listed():
    return [
        # the smallest calls: a quick-look shot on a test-sized model (launch latency counts)
        _prop("model-small", "model", 40, 44, 42, 8, 120, 1, 1, 10, fmax=60.0, host=True),
        # plain single-shot modeling of the 101^3 model with a 50-cell boundary (fields fit the L2)
        _prop("model-101", "model", 101, 101, 101, 50, 1001, 1, 1, 2),
        # a trial model's misfit in the 301 x 301 x 151 inversion, one batch of its shots
        _prop("misfit-301", "misfit", 151, 301, 301, 50, 201, 4, 4, 2, fmax=24.0),
        # a single odd-sized shot migrated from host data through a caller's pad
        _prop("rtm-odd-single", "rtm", 121, 97, 75, 13, 301, 1, 1, 3, host=True),
        # batched migration of the 201^3 model, each shot through its own random pad (the largest)
        _prop("rtm-201-batch", "rtm", 201, 201, 201, 50, 301, 4, 4, 1, pad="shot"),
        # gradients of the small inversion problems, more shots than slots (a ragged last batch)
        _prop("gradient-48-batch", "gradient", 48, 48, 48, 20, 400, 4, 6, 2),
        # the gradient of a preconditioner training model (128^3, nine shots together)
        _prop("gradient-128", "gradient", 128, 128, 128, 50, 151, 9, 9, 2, pad="shot"),
        # the gradient of the 401 x 401 x 201 model at 12.5 m
        _prop("gradient-401", "gradient", 201, 401, 401, 41, 101, 2, 2, 2, dh=12.5, pad="shot"),
        # the misfit of one recorded shot of the 301 x 301 x 151 inversion (22,801 receivers, 2001 samples)
        dict(name="residual-shot", kind="residual", n=22801 * 2001),
        # the finished image of the 201^3 migration, from accumulators summed over GPUs
        dict(name="post-201", kind="post", nz=201, nx=201, ny=201, nb=50, dh=10.0),
        # the learned update of one iteration of the 301 x 301 x 151 inversion
        dict(name="cnn-forward-301", kind="cnn_forward", nz=151, nx=301, ny=301),
        # one training step of the preconditioner on a 128^3 pair
        dict(name="cnn-train-128", kind="cnn_train", nz=128, nx=128, ny=128),
    ]


def _padded(c):
    return tuple(c[k] + 2 * c["nb"] for k in ("nz", "nx", "ny"))


def _tlag(c):
    # the wavelet's delay in samples, as the modeling defines it (FP32)
    t0 = np.float32(2.0) * np.sqrt(np.float32(math.pi)) / np.float32(c["fmax"])
    return int(t0 / np.float32(c["dt"])) + 1


def _updates(c):
    """Field updates of one pass (cells x steps x shots x fields)."""
    n = math.prod(_padded(c)) * (_tlag(c) + c["nt"]) * c["shots"]
    return n * (1 if c["kind"] in ("model", "misfit") else 3)


def draw(rng):
    kind = rng.choice(["model", "model", "misfit", "rtm", "rtm", "gradient", "gradient", "residual", "post",
                       "cnn_forward", "cnn_train"])

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "residual":
        return dict(kind=kind, n=size(1000, 60_000_000) | 1)
    if kind == "post":
        return dict(kind=kind, nz=size(24, 240), nx=size(24, 300), ny=size(24, 300), nb=rng.randint(8, 50), dh=10.0)
    if kind.startswith("cnn"):
        hi = 200 if kind == "cnn_forward" else 140
        return dict(kind=kind, nz=size(24, hi), nx=size(24, hi), ny=size(24, hi))
    batch = rng.randint(1, 5)
    c = _prop("", kind, size(30, 220), size(30, 320), size(30, 320), rng.randint(8, 50), size(60, 600), batch,
              max(1, batch + rng.choice([0, 0, 0, 1, -1])), rng.randint(1, 4), dh=rng.choice([10.0, 12.5]),
              fmax=rng.choice([24.0, 30.0, 60.0]), host=rng.random() < 0.3)
    if kind in ("rtm", "gradient") and rng.random() < 0.5:
        c["pad"] = "shot"
    del c["name"]
    cap = 0.6 * _updates(listed()[4])
    while _updates(c) > cap:
        if c["nt"] > 120:
            c["nt"] = c["nt"] * 2 // 3
        elif c["shots"] > 1:
            c["shots"] -= 1
            c["batch"] = min(c["batch"], c["shots"])
        else:
            c["nx"], c["ny"] = c["nx"] * 3 // 4, c["ny"] * 3 // 4
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _velocity(c, g):
    """Layers with velocities U(1500, 3500) m/s increasing downwards and two
    +-12 % Gaussian anomalies, (ny, nx, nz)."""
    nz, nx, ny = c["nz"], c["nx"], c["ny"]
    u = torch.rand(20, generator=g, device="cuda", dtype=torch.float64)
    vels = torch.sort(1500.0 + 2000.0 * u[:6]).values
    tops = torch.sort(0.08 + 0.84 * u[6:11]).values * nz
    z = torch.arange(nz, device="cuda", dtype=torch.float64)
    v = vels[torch.bucketize(z, tops)].expand(ny, nx, nz).clone()
    ax = [torch.arange(n, device="cuda", dtype=torch.float64) for n in (ny, nx, nz)]
    for k, s in ((11, 0.12), (15, -0.12)):
        sig = (0.06 + 0.1 * float(u[k + 3])) * min(nz, nx, ny)
        e = [torch.exp(-(a - (0.2 + 0.6 * float(u[k + i])) * len(a)) ** 2 / (2 * sig * sig)) for i, a in enumerate(ax)]
        v *= 1.0 + s * e[0][:, None, None] * e[1][None, :, None] * e[2][None, None, :]
    return v.float()


def _pad_given(c, v, g):
    """Edge replication, perturbed by up to 30 % towards the outer faces and
    kept below the leapfrog stability limit."""
    nb = c["nb"]
    p = torch.nn.functional.pad(v[None, None], (nb,) * 6, mode="replicate")[0, 0]
    d = []
    for n in p.shape:
        i = torch.arange(n, device="cuda")
        d.append(torch.clamp(torch.maximum(nb - i, i - (n - 1 - nb)), min=0).float() / nb)
    ramp = torch.maximum(torch.maximum(d[0][:, None, None], d[1][None, :, None]), d[2][None, None, :])
    p = p * (1.0 + 0.3 * ramp * (2.0 * torch.rand(p.shape, generator=g, device="cuda") - 1.0))
    limit = 2.0 / math.sqrt(3.0 * (W[0] + 2.0 * sum(abs(x) for x in W[1:]))) * c["dh"] / c["dt"]
    return torch.clamp(p, max=0.98 * limit)


def _geometry(c, seed):
    """Shots spread over the surface, receivers every `rec` cells, both one
    cell deep; coordinates in metres."""
    rng = np.random.default_rng(seed)
    dh, n = c["dh"], c["shots"]
    side = int(math.ceil(math.sqrt(n)))
    k = np.arange(n)
    u = np.stack([(k % side + 0.5) / side, (k // side + 0.5) / side], 1) + rng.uniform(-0.1, 0.1, (n, 2)) / side
    src = np.stack([u[:, 0] * (c["nx"] - 1) * dh, u[:, 1] * (c["ny"] - 1) * dh, np.full(n, dh)], 1)
    xs, ys = np.arange(0, c["nx"], c["rec"]) * dh, np.arange(0, c["ny"], c["rec"]) * dh
    X, Y = np.meshgrid(xs, ys)
    rec = np.stack([X.ravel(), Y.ravel(), np.full(X.size, dh)], 1)
    return src.astype(np.float32), rec.astype(np.float32)


def _gathers(c, src, rec, g):
    """Recorded data [shot][receiver][nt]: five reflections per shot with
    hyperbolic moveout and Ricker wavelets, and 1 % noise."""
    nt, dt, f = c["nt"], c["dt"], c["fmax"] / 3.0
    r = torch.from_numpy(rec).cuda()
    t = torch.arange(nt, device="cuda") * dt
    out = torch.empty(len(src), len(rec), nt, device="cuda")
    for s in range(len(src)):
        off = ((r[:, :2] - torch.from_numpy(src[s, :2]).cuda()) ** 2).sum(1)
        u = torch.rand(5, 3, generator=g, device="cuda")
        d = out[s]
        d.normal_(generator=g).mul_(0.01)
        for k in range(5):
            t0, v = float(u[k, 0]) * nt * dt, 1500.0 + 1500.0 * float(u[k, 1])
            a = (math.pi * f) ** 2 * (t[None, :] - torch.sqrt(t0 * t0 + off[:, None] / v ** 2)) ** 2
            d.add_((1.0 - 2.0 * a) * torch.exp(-a), alpha=2.0 * float(u[k, 2]) - 1.0)
    return out


def _smooth(shape, g):
    """Random volumes with structure over several cells and some noise."""
    low = torch.randn(1, 3, *[max(2, n // 8) for n in shape], generator=g, device="cuda")
    x = torch.nn.functional.interpolate(low, size=shape, mode="trilinear", align_corners=True)[0]
    return (x + 0.1 * torch.randn(x.shape, generator=g, device="cuda")).contiguous()


def _weights(g):
    """He-scaled weights [4][27][16 out][16 in] and small biases; unused
    channels of the first and last layer are zero."""
    w, b = torch.zeros(4, 27, 16, 16, device="cuda"), torch.zeros(4, 16, device="cuda")
    for k, (ci, co) in enumerate(((3, 16), (16, 16), (16, 16), (16, 1))):
        w[k, :, :co, :ci] = torch.randn(27, co, ci, generator=g, device="cuda") * math.sqrt(2.0 / (27 * ci))
        b[k, :co] = 0.05 * torch.randn(co, generator=g, device="cuda")
    return w, b


def _inputs(c, seed):
    """What prepare() hands to the library and exact() computes from."""
    g = _gen(seed)
    k = c["kind"]
    if k == "residual":
        obs = torch.randn(c["n"], generator=g, device="cuda")
        return dict(obs=obs, cal=0.9 * obs + 0.1 * torch.randn(c["n"], generator=g, device="cuda"))
    if k == "post":
        nzz, nxx, nyy = _padded(c)
        ill = torch.exp(torch.randn(nyy, nxx, nzz, generator=g, device="cuda"))
        return dict(img=_smooth((nyy, nxx, nzz), g)[0] * ill, ill=ill)
    if k.startswith("cnn"):
        shape = (c["ny"], c["nx"], c["nz"])
        w, b = _weights(g)
        return dict(x=_smooth(shape, g), y=_smooth(shape, g)[0].contiguous(), w=w, b=b)
    v = _velocity(c, g)
    src, rec = _geometry(c, seed)
    d = dict(v=v, src=src, rec=rec)
    if k in ("rtm", "gradient"):
        if c["pad"] == "given":
            d["vp"] = _pad_given(c, v, g)
    if k != "model":
        d["data"] = _gathers(c, src, rec, g)
    return d


def prepare(case, seed):
    c = case
    d = _inputs(c, seed)
    k = c["kind"]
    s = dict(c=c)
    if k == "residual":
        s.update(obs=d["obs"], cal=d["cal"], res=torch.empty_like(d["obs"]))
        s["ctx"] = lib.Context(8, 8, 8, 4, 10.0, 8, 1e-3, 30.0)
    elif k == "post":
        s.update(img=d["img"], ill=d["ill"], out=torch.empty(c["ny"], c["nx"], c["nz"], pin_memory=True))
        s["ctx"] = lib.Context(c["nz"], c["nx"], c["ny"], c["nb"], c["dh"], 8, 1e-3, 30.0, lib.BOUNDARY_RBC)
    elif k.startswith("cnn"):
        s.update(x=d["x"], y=d["y"], out=torch.empty_like(d["y"]), net=lib.Cnn(0))
        s["net"].set_weights(d["w"].cpu().numpy(), d["b"].cpu().numpy())
    else:
        back = k in ("rtm", "gradient")
        flags = lib.FLAG_GRAD_DY | lib.FLAG_SUBTRACT_SOURCE if k == "gradient" else 0
        ctx = lib.Context(c["nz"], c["nx"], c["ny"], c["nb"], c["dh"], c["nt"], c["dt"], c["fmax"],
                          lib.BOUNDARY_RBC if back else lib.BOUNDARY_ABC, 0.0 if back else 0.004, c["batch"], flags)
        ctx.set_geometry(d["src"], d["rec"])
        v = d["v"].cpu().numpy()
        if back and c["pad"] == "given":
            ctx.set_padded_velocity(d["vp"].cpu().numpy())
        else:
            ctx.set_velocity(v)
        s.update(ctx=ctx, v=v, shots=list(range(c["shots"])), seed=int(seed) % 1000003)
        n = c["shots"] * len(d["rec"]) * c["nt"]
        if k == "model" and not c["host"]:
            s["out"] = torch.empty(n, device="cuda")
        if k == "misfit":
            s.update(obs=d["data"].reshape(-1), cal=torch.empty(n, device="cuda"), res=torch.empty(n, device="cuda"))
        if back:
            s["data"] = d["data"].cpu().numpy() if c["host"] else d["data"]
            s["img"] = torch.empty(ctx.padded_shape, device="cuda")
            s["ill"] = torch.empty(ctx.padded_shape, device="cuda")
            if c["pad"] == "shot" and k == "rtm":
                ctx.set_shot_random_boundary(kind=0, ratio=100.0, varVp=1000.0, base_seed=s["seed"])
    torch.cuda.synchronize()  # the library runs on streams of its own
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    s, c = state, state["c"]
    k = c["kind"]
    if k == "residual":
        f = s["ctx"].residual_dev(s["obs"].data_ptr(), s["cal"].data_ptr(), c["n"], s["res"].data_ptr())
        return dict(sum=f, residual=s["res"])
    if k == "post":
        s["ctx"].set_accumulators_dev(s["img"].data_ptr(), s["ill"].data_ptr())
        s["ctx"].rtm_image(out=s["out"].numpy())
        return s["out"]
    if k == "cnn_forward":
        s["net"].forward((c["nz"], c["nx"], c["ny"]), s["x"].data_ptr(), s["out"].data_ptr())
        return s["out"]
    if k == "cnn_train":
        loss, gw, gb = s["net"].train_step((c["nz"], c["nx"], c["ny"]), s["x"].data_ptr(), s["y"].data_ptr(), 1e-3,
                                           want_grads=True)
        return dict(loss=loss, gw=gw, gb=gb)
    ctx = s["ctx"]
    if k == "model":
        if c["host"]:
            return ctx.model_shots(s["shots"])
        ctx.model_shots_dev(s["shots"], s["out"].data_ptr())
        return s["out"]
    if k == "misfit":
        ctx.set_velocity(s["v"])
        ctx.model_shots_dev(s["shots"], s["cal"].data_ptr())
        f = ctx.residual_dev(s["obs"].data_ptr(), s["cal"].data_ptr(), s["cal"].numel(), s["res"].data_ptr())
        return dict(misfit=f, cal=s["cal"], residual=s["res"])
    ctx.reset_accumulators()
    if k == "gradient" and c["pad"] == "shot":
        ctx.set_velocity(s["v"])  # each gradient has a new model and new pads
        ctx.set_shot_random_boundary(kind=0, ratio=100.0, varVp=1000.0, base_seed=s["seed"])
    if c["host"]:
        (ctx.rtm_shots if k == "rtm" else ctx.gradient_shots)(s["shots"], s["data"])
        img, ill = ctx.get_accumulators()
    else:
        (ctx.rtm_shots_dev if k == "rtm" else ctx.gradient_shots_dev)(s["shots"], s["data"].data_ptr())
        ctx.get_accumulators_dev(s["img"].data_ptr(), s["ill"].data_ptr())
        img, ill = s["img"], s["ill"]
    return dict(image=img, illumination=ill)


def work(case):
    """Bytes: each time step reads and writes its fields once (two levels and
    the velocity, 16 B a cell; 28 B for the two fields of the fused backward
    step and 16 B for each accumulated cell), data in and results out once.
    FLOPs: 33 a field update (20 additions of the taps at equal distance, five
    multiply-adds, two of the leapfrog)."""
    c = case
    k = c["kind"]
    if k == "residual":
        return dict(bytes=12.0 * c["n"], flops=3.0 * c["n"])
    if k == "post":
        n, m = math.prod(_padded(c)), c["nz"] * c["nx"] * c["ny"]
        return dict(bytes=8.0 * n + 4.0 * m, flops=6.0 * m)
    if k.startswith("cnn"):
        m = c["nz"] * c["nx"] * c["ny"]
        f = 2.0 * 27 * (3 * 16 + 2 * 16 * 16 + 16) * m
        if k == "cnn_forward":
            return dict(bytes=16.0 * m, flops=f)
        return dict(bytes=16.0 * m, flops=3 * f - 2.0 * 27 * 48 * m)
    cells, steps = math.prod(_padded(c)), _tlag(c) + c["nt"]
    data = 4.0 * c["shots"] * c["nt"] * -(-c["nx"] // c["rec"]) * -(-c["ny"] // c["rec"])
    b = 16.0 * cells * steps * c["shots"]
    if k in ("rtm", "gradient"):
        b += (28.0 * cells + 16.0 * c["nz"] * c["nx"] * c["ny"]) * steps * c["shots"] + 8.0 * cells
    return dict(bytes=b + data * (3 if k == "misfit" else 1), flops=33.0 * _updates(c))


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
class _Exact:
    def __init__(self, c, vp, damp=None):
        self.c = c
        f32 = lambda x: float(np.float32(x))  # noqa: E731  (the library takes FP32 parameters)
        self.dt, self.dh = f32(c["dt"]), f32(c["dh"])
        self.v2 = vp.double() ** 2
        self.cv = (self.v2 * (self.dt / self.dh) ** 2)[4:-4, 4:-4, 4:-4].contiguous()
        self.damp = damp
        self.shape = vp.shape
        self.nt, self.tlag = c["nt"], _tlag(c)
        t0, fc = 2.0 * math.sqrt(math.pi) / f32(c["fmax"]), f32(c["fmax"]) / (3.0 * math.sqrt(math.pi))
        a = math.pi ** 3 * fc ** 2 * (np.arange(self.nt) * self.dt - t0) ** 2
        self.w = 1e5 * (1.0 - 2.0 * a) * np.exp(-a) / self.dh ** 3

    def cell(self, p):
        dh, nb = np.float32(self.c["dh"]), self.c["nb"]
        x, y, z = (int((np.float32(q) + np.float32(0.5) * dh) / dh) + nb for q in p)
        return y, x, z

    def cells(self, rec):
        r = np.array([self.cell(p) for p in rec])
        return tuple(torch.from_numpy(r[:, i]).cuda() for i in range(3))

    def lap(self, a):
        n = a.shape
        mid = [slice(4, m - 4) for m in n]
        out = a[mid[0], mid[1], mid[2]] * (-3.0 * W[0])
        for m in range(1, 5):
            for ax in range(3):
                for d in (-m, m):
                    s = list(mid)
                    s[ax] = slice(4 + d, n[ax] - 4 + d)
                    out.add_(a[s[0], s[1], s[2]], alpha=W[m])
        return out

    def step(self, a, q, lap=None):
        """q <- 2a - q + cv lap(a) on the updated cells."""
        i = (slice(4, -4),) * 3
        lap = self.lap(a) if lap is None else lap
        if self.damp is not None:
            q.mul_(self.damp)
        q[i] = torch.addcmul(2.0 * a[i] - q[i], self.cv, lap)
        if self.damp is not None:
            q.mul_(self.damp)

    def forward(self, src, rec=None):
        a = torch.zeros(self.shape, device="cuda", dtype=torch.float64)
        q = torch.zeros_like(a)
        s = self.cell(src)
        a[s] += float(self.w[0])
        seis = torch.zeros(self.nt, len(rec[0]) if rec else 0, device="cuda", dtype=torch.float64)
        for t in range(self.nt + self.tlag):
            if rec and t > self.tlag:
                r = a[rec]
                seis[t - self.tlag] = r if self.damp is None else r * self.damp[rec]
            self.step(a, q)
            if t + 1 < self.nt:
                q[s] += float(self.w[t + 1])
            a, q = q, a
        return seis, a, q

    def backward(self, src, rec, data, u, uold, img, ill, grad):
        """u, uold: the last two forward fields; adds to img and ill."""
        nb, n = self.c["nb"], self.nt + self.tlag
        box = (slice(nb, -nb),) * 3
        off = tuple(slice(nb - 4, m - nb - 4) for m in self.shape)
        s = self.cell(src)
        d = data.double().t().contiguous() / self.dh ** 3
        pr, prold = torch.zeros_like(u), torch.zeros_like(u)
        ps, psold = u, uold
        for t in range(n):
            if t < self.nt:
                pr.index_put_(rec, d[self.nt - 1 - t], accumulate=True)
            lap = self.lap(psold)
            self.step(psold, ps, lap)
            if grad and n - t < self.nt:
                ps[s] += float(self.w[n - t])
            ill[box] += ps[box] ** 2
            if grad:
                img[box] += (self.dt / self.dh ** 2) * pr[box] * lap[off] * self.v2[box]
            else:
                img[box] += ps[box] * pr[box]
            self.step(pr, prold)
            ps, psold, pr, prold = psold, ps, prold, pr


def _damper(c):
    nb, f = c["nb"], float(np.float32(0.004))
    ax = []
    for n in (c["ny"], c["nx"], c["nz"]):
        i = torch.arange(n + 2 * nb, device="cuda", dtype=torch.float64)
        d = torch.minimum(i, n + 2 * nb - 1 - i)
        ax.append((d < nb, torch.where(d < nb, torch.exp(-(f * (nb - d)) ** 2), 0.0)))
    sh = ((slice(None), None, None), (None, slice(None), None), (None, None, slice(None)))
    k = sum(m[s].int() for (m, _), s in zip(ax, sh))
    b = sum(v[s] for (_, v), s in zip(ax, sh))
    return torch.where(k == 0, 1.0, torch.where(k == 1, b, torch.where(k == 2, b - 1.0, 2.0 * b - 5.0)))


def _conv(x, w, b):
    """x (ny, nx, nz, ci), w [27][co][ci], tap t = (dz+1) + 3 (dx+1) + 9 (dy+1)."""
    ny, nx, nz, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = b.expand(ny, nx, nz, len(b))
    for t in range(27):
        z, j, k = t % 3, t // 3 % 3, t // 9
        y = y + p[k:k + ny, j:j + nx, z:z + nz] @ w[t].t()
    return y


def exact(case, seed):
    c = case
    k = c["kind"]
    if k in ("rtm", "gradient") and c["pad"] == "shot":
        return None  # the pads come from the library's own generator
    if k in ("model", "misfit", "rtm", "gradient") and _updates(c) > 8e10:
        return None  # too long in 64 bits
    d = _inputs(c, seed)
    if k == "residual":
        r = d["obs"].double() - d["cal"].double()
        return dict(sum=float((r * r).sum()), residual=r)
    if k == "post":
        nb = c["nb"]
        q = (d["img"].double() / d["ill"].double())[nb:-nb, nb:-nb, nb:-nb]
        out = torch.zeros_like(q)
        out[..., 1:-1] = -(q[..., :-2] - 2.0 * q[..., 1:-1] + q[..., 2:]) / c["dh"] ** 2
        return out
    if k.startswith("cnn"):
        ci, co = (3, 16, 16, 16), (16, 16, 16, 1)
        w = [d["w"][i, :, :co[i], :ci[i]].double().requires_grad_(k == "cnn_train") for i in range(4)]
        b = [d["b"][i, :co[i]].double().requires_grad_(k == "cnn_train") for i in range(4)]
        with torch.set_grad_enabled(k == "cnn_train"):
            x = torch.movedim(d["x"].double(), 0, -1)
            for i in range(4):
                x = _conv(x, w[i], b[i])
                x = torch.relu(x) if i < 3 else x
            if k == "cnn_forward":
                return x[..., 0]
            loss = 0.5 * ((x[..., 0] - d["y"].double()) ** 2).mean()
            loss.backward()
        gw, gb = torch.zeros(4, 27, 16, 16, dtype=torch.float64), torch.zeros(4, 16, dtype=torch.float64)
        for i in range(4):
            gw[i, :, :co[i], :ci[i]] = w[i].grad.cpu()
            gb[i, :co[i]] = b[i].grad.cpu()
        return dict(loss=float(loss.detach()), gw=gw, gb=gb)
    if k in ("model", "misfit"):
        nb = c["nb"]
        vp = torch.nn.functional.pad(d["v"][None, None], (nb,) * 6, mode="replicate")[0, 0]
        e = _Exact(c, vp, _damper(c))
        rec = e.cells(d["rec"])
        seis = [e.forward(src, rec)[0].t().contiguous() for src in d["src"]]
        if k == "model":
            return seis if c["host"] else torch.stack(seis).reshape(-1)
        cal = torch.stack(seis).reshape(-1)
        r = d["data"].reshape(-1).double() - cal
        return dict(misfit=float((r * r).sum()), cal=cal, residual=r)
    e = _Exact(c, d["vp"])
    rec = e.cells(d["rec"])
    img = torch.zeros(e.shape, device="cuda", dtype=torch.float64)
    ill = torch.zeros_like(img)
    for i, src in enumerate(d["src"]):
        _, u, uold = e.forward(src)
        e.backward(src, rec, d["data"][i], u, uold, img, ill, k == "gradient")
    return dict(image=img, illumination=ill)
