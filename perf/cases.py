"""The work that programs built on this framework have it do, as cases that
can be measured: modelling, gradients of the misfit (exact and by the imaging
condition), and the learned preconditioner's network, each through its public
entry points, from a single shot on a toy grid to a batch of shots on a
608 x 2000 model.

``exact`` restates the physics in plain torch in 64 bits: a derivative is a
product with a banded matrix whose rows hold exactly the stencil terms that
the staggered scheme forms there, so autograd gives the exact gradient.
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

from stfwi_b200 import Solver
from stfwi_b200.autograd import elastic_forward, elastic_misfit
from stfwi_b200.learned.unet import HEAD_IN, LAYERS, UNet, padded_shape

GRID = dict(pad=20, fd=8, surface=True, shots=1, source="mix", density=False, segment=0, tune=False)


def listed():
    def grid(name, kind, nz, nx, steps, **kw):
        return {**GRID, "name": name, "kind": kind, "nz": nz, "nx": nx, "steps": steps, **kw}

    return [
        # the smallest call: a gradient check on a toy grid, launch latency throughout
        grid("check_24x32_fd2", "misfit", 24, 32, 60, pad=8, fd=2, surface=False, source="moment"),
        # modelling one shot, as an interactive user does
        grid("model_1shot_152x500_fd8", "model", 152, 500, 1000, source="force"),
        # the single-shot gradient of a Marmousi-sized model, every step kept
        grid("misfit_1shot_152x500_fd4", "misfit", 152, 500, 2000, fd=4, source="force"),
        # ragged sizes, absorbing on all sides, a loss of the user's own on all four components
        grid("traces_13shots_97x333_fd4", "traces", 97, 333, 300, pad=11, fd=4, surface=False, shots=13),
        # all three parameters inverted: the history also holds the velocities
        grid("density_10shots_152x500_fd8", "misfit", 152, 500, 400, shots=10, density=True),
        # the imaging-condition backend
        grid("imaging_10shots_152x500_fd8", "imaging", 152, 500, 400, shots=10),
        # the batched gradient that an inversion repeats, with its tuned schedule
        grid("misfit_50shots_152x500_fd8", "misfit", 152, 500, 500, shots=50, tune=True),
        # observed data made for a whole survey
        grid("model_34shots_152x500_fd8", "model", 152, 500, 500, shots=34),
        # the middle grid of an uneven batch, default schedule
        grid("misfit_16shots_304x1000_fd8", "misfit", 304, 1000, 200, shots=16),
        # the largest grid, with a history that has to be checkpointed
        grid("segments_32shots_608x2000_fd8", "misfit", 608, 2000, 100, shots=32, segment=40),
        # one learned step of an inversion: the network on one model's features
        {"name": "net_1x152x500", "kind": "net", "nz": 152, "nx": 500, "batch": 1},
        # a training batch: forward, loss and all gradients
        {"name": "train_8x152x500", "kind": "train", "nz": 152, "nx": 500, "batch": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["misfit", "misfit", "misfit", "model", "model", "traces", "imaging", "net", "train"])
    if kind in ("net", "train"):
        return {"kind": kind, "nz": rng.randint(60, 320), "nx": rng.randint(200, 1020), "batch": _log(rng, 1, 12)}
    while True:
        nz = _log(rng, 24, 608)
        nx = min(2000, max(32, int(nz * rng.uniform(1.2, 4.0))))
        c = dict(GRID, kind=kind, nz=nz, nx=nx, steps=_log(rng, 60, 1500), shots=_log(rng, 1, 50),
                 fd=rng.choice([2, 4, 8, 8]), surface=rng.random() < 0.7, pad=rng.choice([8, 11, 16, 20, 20, 20, 30]),
                 source=rng.choice(["force", "moment", "mix"]))
        if kind == "misfit":
            c["density"] = rng.random() < 0.25
            c["segment"] = rng.choice([0, 0, 0, max(10, c["steps"] // rng.randint(3, 9))])
            c["tune"] = c["shots"] >= 8 and rng.random() < 0.3
        kept = (c["segment"] or c["steps"]) if kind != "model" else 1
        if _cells(c) * c["shots"] * c["steps"] < 3e9 and kept * c["shots"] * nz * nx * (20 if c["density"] else 12) < 25e9:
            return c


# ----------------------------------------------------------------- inputs


def _cells(c):
    return (c["nz"] + c["pad"] * (1 if c["surface"] else 2)) * (c["nx"] + 2 * c["pad"])


def _spacing(c):
    dx = 20.0 if c["nz"] < 300 else 10.0 if c["nz"] < 600 else 5.0
    return dx, 7.5e-5 * dx, 100.0 / dx      # metres, seconds, peak frequency


def _earth(c, seed):
    """(Vs, Vp, rho): layers whose velocity grows with depth, dipping and smoothly disturbed."""
    rng = np.random.default_rng(seed)
    nz, nx = c["nz"], c["nx"]
    z, x = np.arange(nz)[:, None] / nz, np.arange(nx)[None, :] / nx
    depth = z + rng.uniform(-0.1, 0.1) * x
    for _ in range(4):
        depth = depth + 0.02 * np.sin(2 * np.pi * (rng.uniform(0.5, 4) * x + rng.uniform(0.5, 3) * z + rng.uniform()))
    tops = np.sort(rng.uniform(0.05, 0.95, 9))
    layer = sum((depth > t).astype(np.int64) for t in tops)
    vp = np.linspace(1600.0, 4200.0, 10)[layer] + rng.uniform(-100, 100, 10)[layer] + 200.0 * (depth - 0.5)
    vp = np.clip(vp, 1500.0, 4700.0)
    vs = np.clip(vp / rng.uniform(1.6, 2.0, 10)[layer], 800.0, 2750.0)
    rho = np.clip(310.0 * vp ** 0.25, 1700.0, 2600.0)
    return tuple(torch.from_numpy(a.astype(np.float32)).cuda() for a in (vs, vp, rho))


def _ricker(t, f):
    a = (math.pi * f * t) ** 2
    return (1.0 - 2.0 * a) * torch.exp(-a)


def _survey(c, seed):
    """Sources (x, z, type), their wavelets, receivers, and observed traces
    [shots, steps, receivers]: direct arrivals of a seeded medium and noise."""
    dx, dt, fc = _spacing(c)
    g = torch.Generator(device="cuda").manual_seed(seed)
    ns, nt = c["shots"], c["steps"]
    first = int(torch.randint(0, c["nx"], (1,), generator=g, device="cuda"))
    sx = (first + np.arange(ns) * max(1, c["nx"] // ns)) % c["nx"]
    sz = np.full(ns, min(2, c["nz"] - 1))
    types = ["force", "moment"] * ((ns + 1) // 2) if c["source"] == "mix" else [c["source"]] * ns
    types = types[:ns]
    rx = np.arange(0, c["nx"], 2, dtype=np.int32)
    rz = np.ones_like(rx)
    t = torch.arange(nt, device="cuda", dtype=torch.float64) * dt
    # an explosion's moment that radiates velocities of the force's order
    amp = torch.tensor([3000.0 if k == "moment" else 1.0 for k in types], device="cuda", dtype=torch.float64)
    f = fc * (0.9 + 0.2 * torch.rand(ns, 1, generator=g, device="cuda", dtype=torch.float64))
    wav = (amp[:, None] * _ricker(t[None] - 1.5 / fc, f)).float()
    dist = dx * (torch.from_numpy(rx).cuda()[None] - torch.from_numpy(sx).cuda()[:, None]).abs().double()
    late = 1.7 / fc + dist / (1500.0 + 500.0 * torch.rand(ns, 1, generator=g, device="cuda", dtype=torch.float64))
    size = 8.0 * dt / (dx * dx * 2000.0) / torch.sqrt(1.0 + dist / dx)
    obs = size[:, None] * _ricker(t[None, :, None] - late[:, None], fc)
    obs = obs + 0.02 * size.mean() * torch.randn(obs.shape, generator=g, device="cuda", dtype=torch.float64)
    return sx, sz, types, wav, rx, rz, obs.float()


def _lowpass(fcut, dt):
    """Sixth-order Butterworth low-pass as second-order sections (bilinear transform)."""
    w, out = math.tan(math.pi * min(fcut * dt, 0.45)), []
    for k in range(3):
        a = 2.0 * math.sin(math.pi * (2 * k + 1) / 12.0) * w
        n = 1.0 + a + w * w
        out.append([w * w / n, 2 * w * w / n, w * w / n, 1.0, 2 * (w * w - 1) / n, (1 - a + w * w) / n])
    return np.array(out)


def _net_inputs(c, seed):
    """Features [gradient, illumination, Vp, Vs] scaled as the network is fed
    them, a target update, and the weight of each pixel (0 outside the model)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    h, w = padded_shape(c["nz"], c["nx"])
    b, nz, nx = c["batch"], c["nz"], c["nx"]
    raw = torch.randn(b, 5, nz // 8 + 2, nx // 8 + 2, generator=g, device="cuda")
    maps = torch.nn.functional.interpolate(raw, size=(nz, nx), mode="bilinear", align_corners=False)
    feat = maps[:, :4].contiguous()
    target, weight = torch.zeros(b, h, w, device="cuda"), torch.zeros(b, h, w, device="cuda")
    target[:, :nz, :nx], weight[:, :nz, :nx] = 0.3 * maps[:, 4], 1.0
    return h, w, feat, target, weight


def prepare(case, seed):
    c = case
    if c["kind"] in ("net", "train"):
        h, w, feat, target, weight = _net_inputs(c, seed)
        return {"kind": c["kind"], "net": UNet(h, w, seed=seed), "feat": feat, "target": target, "weight": weight,
                "norm": 1.0 / float(weight.sum())}
    dx, dt, fc = _spacing(c)
    sx, sz, types, wav, rx, rz, obs = _survey(c, seed)
    vs, vp, rho = _earth(c, seed)
    solver = Solver(c["nz"], c["nx"], dx, dx, dt, c["steps"], fc, c["pad"], len(rx), c["shots"], fd_order=c["fd"],
                    free_surface=c["surface"], want_gradient=c["kind"] != "model", density=c["density"],
                    ckpt_interval=c["segment"])
    solver.set_receivers(rx, rz)
    solver.set_shots(sx, sz, types, wav)
    if c["tune"]:
        solver.set_model(vs, vp, rho)
        solver.autotune(steps=10)
    s = {"kind": c["kind"], "solver": solver, "vs": vs, "vp": vp, "rho": rho, "obs": obs, "density": c["density"]}
    if c["kind"] == "model":
        s["rec"] = torch.empty((c["shots"], 4, c["steps"], len(rx)), device="cuda")
    else:
        s["scale"] = float(1.0 / obs.double().square().mean())
        s["sos"], s["taper"] = _lowpass(0.6 * fc, dt), c["steps"] // 10
    return s


# ----------------------------------------------------------------- one pass


def run(state):
    s = state
    if s["kind"] == "net":
        return s["net"].forward(s["net"].pack(s["feat"]))
    if s["kind"] == "train":
        net = s["net"]
        x = net.pack(s["feat"])
        net.zero_grad()
        net.forward(x, train=True)
        net.backward(x, s["target"], s["weight"], s["norm"])
        return net.grads
    S = s["solver"]
    if s["kind"] == "model":
        S.set_model(s["vs"], s["vp"], s["rho"])
        S.forward()
        return S.records(out=s["rec"])
    if s["kind"] == "imaging":
        # the gradient in the model's type, as a float32 optimizer takes it
        S.set_model(s["vs"], s["vp"], s["rho"])
        S.forward(store=True)
        S.misfit(s["obs"], 1, s["scale"], s["sos"], s["taper"])
        g = torch.empty((1, 3, S.nz_dom, S.nx_dom), dtype=torch.float64, device="cuda")
        S.gradient(exact=False, imaging=True, out=g)
        return g[0].to(s["vs"].dtype)
    vs, vp = s["vs"].detach().requires_grad_(), s["vp"].detach().requires_grad_()
    rho = s["rho"].detach().requires_grad_(s["density"])
    if s["kind"] == "misfit":
        loss = elastic_misfit(vs, vp, rho, S, s["obs"], 1, s["scale"], s["sos"], s["taper"])
        loss.backward()
        out = {"loss": loss.detach().to(vs.dtype), "vs": vs.grad, "vp": vp.grad}
    else:
        traces = elastic_forward(vs, vp, rho, S)
        loss = 0.5 * s["scale"] * (traces[:, 0].square().sum() + (traces[:, 1] - s["obs"]).square().sum()
                                   + 1e6 * traces[:, 2:].square().sum())
        loss.backward()
        out = {"traces": traces.detach(), "vs": vs.grad, "vp": vp.grad}
    if s["density"]:
        out["rho"] = rho.grad
    return out


# ----------------------------------------------------------------- work


def work(case):
    """One step reads the five fields once and writes them once (4 bytes a
    cell each) and writes or reads the three stresses kept for the gradient
    (five fields with the density); eight derivatives of 3 FD/2 operations
    and about 40 more a cell and step.  A checkpointed pass models twice."""
    c = case
    if c["kind"] in ("net", "train"):
        h, w = padded_shape(c["nz"], c["nx"])
        level = {"1": 0, "2": 1, "3": 2}
        flops = sum(2 * 9 * ci * co * (h * w >> 2 * level.get(name[3], 3)) for name, ci, co in LAYERS)
        weights = sum(9 * ci * co for _, ci, co in LAYERS)
        if c["kind"] == "net":
            return {"flops": c["batch"] * flops, "bytes": c["batch"] * (16 * c["nz"] * c["nx"] + 4 * h * w) + 2 * weights}
        acts = sum(2 * co * (h * w >> 2 * level.get(name[3], 3)) for name, ci, co in LAYERS)
        return {"flops": 3 * c["batch"] * flops,
                "bytes": c["batch"] * (16 * c["nz"] * c["nx"] + 8 * h * w + 2 * acts) + 6 * weights}
    cells, phys = c["shots"] * _cells(c), c["shots"] * c["nz"] * c["nx"]
    passes = 1 if c["kind"] == "model" else 3 if c["segment"] else 2
    kept = 0 if c["kind"] == "model" else 2 * (5 if c["density"] else 3)
    rec = 16.0 * c["shots"] * c["steps"] * ((c["nx"] + 1) // 2)
    return {"flops": passes * cells * c["steps"] * (12.0 * c["fd"] + 40.0),
            "bytes": c["steps"] * (passes * cells * 40.0 + kept * phys * 4.0) + rec + 16.0 * c["nz"] * c["nx"]}


# ----------------------------------------------------------------- 64 bits


def _derivatives(n, fd):
    """Forward and backward staggered differences of n samples as banded
    matrices; a term is formed only where both of its samples exist."""
    coef = {2: [1.0], 4: [9 / 8, -1 / 24], 8: [1225 / 1024, -245 / 3072, 49 / 5120, -5 / 7168]}[fd]
    plus = torch.zeros(n, n, dtype=torch.float64)
    for k, v in enumerate(coef, 1):
        t = torch.arange(k - 1, n - k)
        plus[t, t + k] += v
        plus[t, t - k + 1] -= v
    minus = torch.zeros(n, n, dtype=torch.float64)
    minus[1:] = plus[:-1]
    return plus.cuda(), minus.cuda(), coef[0]


def _profile(n, low, high, width, dx, dt, fc, vmax):
    """(b, a, 1/k) of the absorbing layer along one axis: `width` cells at the low and the high end."""
    b, a, ik = np.ones(n), np.zeros(n), np.ones(n)
    length = width * dx
    d0 = np.float32(-3.0) * np.float32(vmax) * np.float32(math.log(1e-3)) / np.float32(2.0 * length)
    for i in range(width):
        r = (i + 1) * dx / length
        d, k, al = float(d0) * r * r, 1.0 + r * r, math.pi * fc * (1.0 - r)
        bb = math.exp(-(d / k + al) * dt)
        den = k * (d + k * al)
        for at in ([width - 1 - i] if low else []) + ([n - width + i] if high else []):
            b[at], a[at], ik[at] = bb, d * (bb - 1.0) / den if den > 1e-10 else 0.0, 1.0 / k
    return [torch.from_numpy(v).cuda() for v in (b, a, ik)]


class _Physics:
    def __init__(self, c, seed):
        self.c = c
        self.dx, self.dt, self.fc = _spacing(c)
        p, self.top = c["pad"], 0 if c["surface"] else c["pad"]
        self.nz, self.nx = c["nz"] + p + self.top, c["nx"] + 2 * p
        self.Xp, self.Xm, self.c1 = _derivatives(self.nx, c["fd"])
        self.Zp, self.Zm, _ = _derivatives(self.nz, c["fd"])
        self.model = [m.double().requires_grad_() for m in _earth(c, seed)]
        vmax = float(self.model[1].max())
        self.px = [v[None, None] for v in _profile(self.nx, True, True, p, self.dx, self.dt, self.fc, vmax)]
        self.pz = [v[None, :, None] for v in _profile(self.nz, not c["surface"], True, p, self.dx, self.dt, self.fc, vmax)]
        sx, sz, types, wav, rx, rz, obs = _survey(c, seed)
        self.wav, self.obs = wav.double(), obs.double()
        self.ix, self.iz = torch.from_numpy(sx + p).cuda(), torch.from_numpy(sz + self.top).cuda()
        self.force = torch.tensor([k == "force" for k in types], device="cuda").double()
        self.rx, self.rz = torch.from_numpy(rx).long().cuda() + p, torch.from_numpy(rz).long().cuda() + self.top
        # rectangles in which the scheme forms its derivatives
        i, j = torch.arange(self.nz, device="cuda")[:, None], torch.arange(self.nx, device="cuda")[None]
        self.vel = ((i < self.nz - 1) & (j > 0) & (j < self.nx - 1)).double()
        self.notleft, self.notright = (j > 0).double() + 0 * i, (j < self.nx - 1).double() + 0 * i
        self.shear = ((i < self.nz - 1) & (j < self.nx - 1)).double()
        self.row0 = (i == 0).double() * (1.0 if c["surface"] else 0.0)

    def embed(self, m):
        """The model on the padded grid; the copies outside it are constants."""
        p, c = self.c["pad"], self.c
        ii = (torch.arange(self.nz, device="cuda") - self.top).clamp(0, c["nz"] - 1)
        jj = (torch.arange(self.nx, device="cuda") - p).clamp(0, c["nx"] - 1)
        wide = m.detach()[ii][:, jj]
        inner = torch.nn.functional.pad(m - m.detach(), (p, p, self.top, p))
        return wide + inner

    def materials(self):
        vs, vp, rho = (self.embed(m) for m in self.model)
        mu, l2m = rho * vs * vs, rho * vp * vp
        return l2m, l2m - 2 * mu, mu, 1.0 / rho

    def steps(self, n0, n1, l2m, lam, mu, b, *carry):
        """Steps [n0, n1); returns the carry and the traces [n1 - n0, 4, shots, receivers]."""
        U, V, sxx, szz, sxz = carry[:5]
        psi, dt, h = list(carry[5:]), self.dt, self.dt / self.dx
        shot = torch.arange(self.c["shots"], device="cuda")
        at = torch.zeros(self.c["shots"], self.nz, self.nx, dtype=torch.float64, device="cuda")
        at[shot, self.iz, self.ix] = 1.0
        lm = (lam + mu)[self.iz, self.ix]
        rec = []

        def absorb(d, k, prof):
            psi[k] = prof[0] * psi[k] + prof[1] * d
            return d * prof[2] + psi[k]

        for n in range(n0, n1):
            dxx = absorb(sxx @ self.Xp.T, 0, self.px)
            dzs = absorb(self.Zm @ sxz * (1 - self.row0) + self.row0 * 2 * self.c1 * sxz, 1, self.pz)
            dxs = absorb(sxz @ self.Xm.T, 2, self.px)
            dzz = absorb(self.Zp @ szz, 3, self.pz)
            U = U + self.vel * b * h * (dxx + dzs)
            V = V + self.vel * b * h * (dxs + dzz) + at * (dt / self.dx ** 2 * self.force * self.wav[:, n])[:, None, None] * b
            dxu = absorb(U @ self.Xm.T, 4, self.px)
            dzv = absorb(self.notright * (self.Zm @ V * (1 - self.row0) - self.row0 * lam / l2m * dxu), 5, self.pz)
            dzu = absorb(self.notleft * (self.Zp @ U), 6, self.pz)
            dxv = absorb(V @ self.Xp.T, 7, self.px)
            boom = at * ((1 - self.force) * self.wav[:, n] * dt / (2 * lm * self.dx ** 2))[:, None, None]
            ex, ez = h * dxu * self.notleft + boom, h * dzv + boom
            sxx, szz = sxx + l2m * ex + lam * ez, szz + lam * ex + l2m * ez
            sxz = sxz + mu * self.shear * h * (dzu + dxv)
            p = (slice(None), self.rz, self.rx)
            det = ((l2m - lam) * (l2m + lam))[p[1:]]
            rec.append(torch.stack([U[p], V[p], (l2m[p[1:]] * sxx[p] - lam[p[1:]] * szz[p]) / det,
                                    (l2m[p[1:]] * szz[p] - lam[p[1:]] * sxx[p]) / det]))
        return (torch.stack(rec), U, V, sxx, szz, sxz, *psi)

    def traces(self, grad):
        """[shots, 4, steps, receivers]"""
        nt, ns = self.c["steps"], self.c["shots"]
        mats = self.materials()
        carry = [torch.zeros(ns, self.nz, self.nx, dtype=torch.float64, device="cuda") for _ in range(13)]
        chunk = max(1, min(50, int(3e10 / (ns * self.nz * self.nx * 8 * 60))))
        out = []
        for n in range(0, nt, chunk):
            args = (n, min(n + chunk, nt), *mats, *carry)
            got = torch.utils.checkpoint.checkpoint(self.steps, *args, use_reentrant=False) if grad else self.steps(*args)
            out.append(got[0])
            carry = got[1:]
        return torch.cat(out).permute(2, 1, 0, 3)


def _cascade(x, sos):
    """Second-order sections along dimension 1 of x [shots, steps, receivers]."""
    for b0, b1, b2, _, a1, a2 in sos:
        z1, z2, y = torch.zeros_like(x[:, 0]), torch.zeros_like(x[:, 0]), torch.empty_like(x)
        for n in range(x.shape[1]):
            v = b0 * x[:, n] + z1
            z1, z2 = b1 * x[:, n] - a1 * v + z2, b2 * x[:, n] - a2 * v
            y[:, n] = v
        x = y
    return x


def _net_exact(c, seed):
    h, w, feat, target, weight = _net_inputs(c, seed)
    net, F = UNet(h, w, seed=seed), torch.nn.functional
    flat = net.params.double().requires_grad_()

    def conv(name, x):
        ci, co = next((i, o) for n, i, o in LAYERS if n == name)
        wo, bo = net.lay[name]
        k = flat[wo:bo].view(3, 3, co, ci).permute(2, 3, 0, 1)
        return torch.relu(F.conv2d(x, k, flat[bo:bo + co], padding=1))

    x = torch.zeros(c["batch"], 16, h, w, dtype=torch.float64, device="cuda")
    x[:, :4, :c["nz"], :c["nx"]] = feat.double()
    skips = []
    for level in "123":
        x = conv("enc%sb" % level, conv("enc%sa" % level, x))
        skips.append(x)
        x = F.avg_pool2d(x, 2)
    x = conv("botb", conv("bota", x))
    for level in "321":
        x = torch.cat([F.interpolate(x, scale_factor=2, mode="nearest"), skips.pop()], 1)
        x = conv("dec%sb" % level, conv("dec%sa" % level, x))
    hw, hb = net.head
    out = torch.einsum("bchw,c->bhw", x, flat[hw:hw + HEAD_IN]) + flat[hb]
    if c["kind"] == "net":
        return out.detach()
    loss = (weight.double() * (out - target.double()).square()).sum() / float(weight.sum())
    return torch.autograd.grad(loss, flat)[0]


def exact(case, seed):
    c = case
    if c["kind"] in ("net", "train"):
        return _net_exact(c, seed)
    if c["kind"] == "imaging":
        return None      # the imaging condition is an approximation of the gradient, not a number of its own
    cost = c["shots"] * _cells(c) * (c["nx"] + c["nz"]) * 8.0 * c["steps"] * (1 if c["kind"] == "model" else 4)
    if cost > 1.5e14 or c["steps"] * (1 if c["kind"] == "model" else 4) > 8000:
        return None      # over about 20 seconds
    P = _Physics(c, seed)
    if c["kind"] == "model":
        with torch.no_grad():
            return P.traces(False)
    tr = P.traces(True)
    scale = float(1.0 / P.obs.square().mean())
    if c["kind"] == "misfit":
        nt, n_taper = c["steps"], c["steps"] // 10
        m = torch.arange(1, n_taper + 1, device="cuda", dtype=torch.float64)
        taper = torch.ones(nt, dtype=torch.float64, device="cuda")
        if n_taper:
            taper[nt - n_taper:] = (torch.cos(m / n_taper * math.pi) + 1.0) / 2.0
        sos = _lowpass(0.6 * P.fc, P.dt)
        with torch.no_grad():
            r = _cascade(taper[None, :, None] * (tr[:, 1] - P.obs), sos)
            loss = scale * r.square().mean()
            cot = taper[None, :, None] * _cascade(r.flip(1), sos).flip(1) * (2.0 * scale / r.numel())
        g = torch.autograd.grad(tr[:, 1], P.model, cot)
        out = {"loss": loss, "vs": g[0], "vp": g[1]}
    else:
        loss = 0.5 * scale * (tr[:, 0].square().sum() + (tr[:, 1] - P.obs).square().sum() + 1e6 * tr[:, 2:].square().sum())
        g = torch.autograd.grad(loss, P.model)
        out = {"traces": tr.detach(), "vs": g[0], "vp": g[1]}
    if c["density"]:
        out["rho"] = g[2]
    return out
