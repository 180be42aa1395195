"""What the framework is asked to do in use, as timed cases.

Every case is one call sequence of the public Python binding (qpstd.py, over
the C ABI of include/qpstd.h) on seeded synthetic shots: time steps of a
resident shot, whole reverse-time migrations, a batch of shots with uneven
windows, a served mix and the one-call form.  exact() restates the equations
in 64 bits with torch FFTs.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "constant-q-pstd_gb300"))
import qpstd  # noqa: E402

PI = 3.1415926  # the value the programs use
DX = 10.0
KINDS = {"aps": qpstd.APS, "vaps": qpstd.VAPS, "artm": qpstd.ARTM, "qrtm": qpstd.QRTM}


def listed():
    return [
        # A short burst of steps on a small window: the latency of a launch and of one line.
        dict(name="aps_small", path="steps", kind="aps", nxx=101, nzz=80, pml=10, nt=60, dt=0.001, rank=0),
        # Acoustic modeling of the 160 x 398 model with CPML 20 (439 is prime), receivers on every column.
        dict(name="aps_439x200", path="steps", kind="aps", nxx=439, nzz=200, pml=20, nt=120, dt=0.001, rank=0),
        # A deep acoustic window of the serving mix (2048 cells down), a smooth width.
        dict(name="aps_deep", path="steps", kind="aps", nxx=800, nzz=2088, pml=20, nt=120, dt=0.0005, rank=0),
        # Constant-Q modeling of the 160 x 398 model.
        dict(name="vaps_439x200", path="steps", kind="vaps", nxx=439, nzz=200, pml=20, nt=80, dt=0.001, rank=0),
        # The same in the low-rank form, rank 4 (one factor per layer velocity).
        dict(name="vaps_lowrank_439x200", path="steps", kind="vaps", nxx=439, nzz=200, pml=20, nt=80, dt=0.001,
             rank=4),
        # One acoustic RTM on a ragged window (both sides odd, the width a prime).
        dict(name="artm_ragged", path="rtm", kind="artm", nxx=337, nzz=251, pml=20, nt=60, dt=0.001, snaps=6,
             eta=1e-20),
        # The large acoustic RTM window: 800 x 2400 model, CPML 30.
        dict(name="artm_2461x860", path="rtm", kind="artm", nxx=2461, nzz=860, pml=30, nt=40, dt=0.0005, snaps=8,
             eta=1e-20),
        # One Q-RTM shot of the batched workload (1678 = 2 * 839).
        dict(name="qrtm_1678x660", path="rtm", kind="qrtm", nxx=1678, nzz=660, pml=30, nt=24, dt=0.0005, snaps=6,
             eta=1e-20),
        # Q-RTM with a stabilisation large enough that the filter changes every step.
        dict(name="qrtm_stabilised", path="rtm", kind="qrtm", nxx=733, nzz=421, pml=20, nt=24, dt=0.0005, snaps=5,
             eta=1e4),
        # Sixteen Q-RTM shots with uneven windows advancing together (600 deep, 600 .. 2000 wide).
        dict(name="qrtm_batch", path="batch", kind="qrtm", nxx=1300, nzz=660, pml=30, nt=12, dt=0.0005, snaps=4,
             eta=1e-20, shots=16),
        # Requests of all four kinds and uneven grids served together from host buffers.
        dict(name="server_mix", path="server", kind="mix", nxx=700, nzz=400, pml=20, nt=60, dt=0.0005, snaps=6,
             eta=1e-20, shots=10),
        # One whole shot through the one-call form, host arrays in, gather out (the programs' serial path).
        dict(name="one_call_vaps", path="call", kind="vaps", nxx=300, nzz=180, pml=10, nt=300, dt=0.001, rank=0),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Windows from 80 to 4136 wide and 60 to 2088 deep, every path and kind."""
    path = rng.choice(["steps", "steps", "steps", "rtm", "rtm", "rtm", "batch", "server", "call"])
    pml = rng.choice([10, 20, 30])
    lo = 2 * pml + 30
    nxx, nzz = _logu(rng, lo, 4136), _logu(rng, lo, 2088)
    dt = rng.choice([0.0005, 0.001])
    budget = 6.0e7  # points x steps of a pass, about half the largest listed case
    c = dict(path=path, nxx=nxx, nzz=nzz, pml=pml, dt=dt)
    if path in ("steps", "call"):
        while nxx * nzz > 2200000:
            nzz = max(lo, nzz // 2)
        nt = max(8, min(rng.choice([40, 80, 160]), int(budget / (nxx * nzz))))
        kind = rng.choice(["aps", "vaps"])
        rank = rng.choice([0, 0, 3, 4, 5]) if kind == "vaps" and path == "steps" else 0
        c.update(kind=kind, nzz=nzz, nt=nt, rank=rank)
    elif path == "rtm":
        while nxx * nzz > 2200000:
            nzz = max(lo, nzz // 2)
        nt = max(8, min(rng.choice([20, 40, 60]), int(budget / (4 * nxx * nzz))))
        c.update(kind=rng.choice(["artm", "qrtm"]), nzz=nzz, nt=nt, snaps=rng.choice([3, 6, 10]),
                 eta=rng.choice([1e-20, 1e-20, 1e4]))
    else:
        shots = rng.randint(4, 16) if path == "batch" else rng.randint(4, 10)
        nxx, nzz = _logu(rng, 150, 1800 if path == "batch" else 700), _logu(rng, 100, 700)
        nt = max(8, min(40, int(budget / (4 * shots * nxx * nzz))))
        c.update(kind=rng.choice(["artm", "qrtm"]) if path == "batch" else "mix", nxx=nxx, nzz=nzz, nt=nt,
                 snaps=rng.choice([3, 5, 8]), eta=1e-20, shots=shots)
    return c


# ---- inputs -----------------------------------------------------------------------
def _wavelet(nt, dt, fd):
    """A Ricker wavelet that starts from zero (its first quarter period is ramped in)."""
    t = np.arange(nt) * dt - 0.5 / fd
    a = (PI * fd * t) ** 2
    ramp = np.minimum(1.0, np.arange(nt) * dt * 4.0 * fd)
    return ((1.0 - 2.0 * a) * np.exp(-a) * ramp).astype(np.float32)


def _shot(kind, nxx, nzz, pml, nt, dt, seed, snaps=0, eta=0.0, layers_only=False):
    """One seeded shot: flat layers plus two anomalies, Gardner density, Q per layer, edges repeated into the CPML."""
    rng = np.random.default_rng(seed)
    nx, nz, fd = nxx - 2 * pml, nzz - 2 * pml, 20.0
    nl = 4 if layers_only else 6
    vel = np.sort(rng.uniform(1500.0, 4200.0, nl))
    layer = np.searchsorted(np.sort(rng.uniform(0, nz, nl - 1)), np.arange(nz), side="right")
    layer = np.pad(layer, pml, mode="edge")
    vp = np.broadcast_to(vel[layer][None, :], (nxx, nzz)).copy()
    if not layers_only:
        x, z = np.arange(nxx), np.arange(nzz)
        for _ in range(2):
            cx, cz, w = rng.uniform(0.2, 0.8) * nxx, rng.uniform(0.3, 0.8) * nzz, rng.uniform(0.03, 0.06) * (nxx + nzz)
            vp += rng.choice([-250.0, 250.0]) * np.outer(np.exp(-((x - cx) / w) ** 2), np.exp(-((z - cz) / w) ** 2))
    rho = 310.0 * np.sqrt(np.sqrt(vp))
    bbx, bbz = 1.0 / rho, 1.0 / rho
    bbx[:-1] = 2.0 / (rho[:-1] + rho[1:])
    bbz[:, :-1] = 2.0 / (rho[:, :-1] + rho[:, 1:])
    d = dict(kind=KINDS[kind], nxx=nxx, nzz=nzz, pml=pml, dx=DX, dz=DX, dt=dt, fd=fd, nt=nt, rik=_wavelet(nt, dt, fd),
             xsg=pml + nx // 2, zsg=pml + 2, gxg=np.arange(pml, pml + nx, dtype=np.int32),
             gzg=np.full(nx, pml + 2, dtype=np.int32), snaps=snaps, etas=eta, etar=eta, taoc=0.0)
    m = dict(vp=vp, rho=rho, bbx=bbx, bbz=bbz)
    if kind in ("vaps", "qrtm"):
        ql = rng.uniform(30.0, 150.0, nl)
        q = ql[layer][None, :]
        gam = np.broadcast_to(1.0 / PI / q, vp.shape)
        m.update(gam=gam, lam=np.ones_like(vp), vwd=np.exp(np.log(vp / (2 * PI * fd)) / 16.0), tao=vp / q)
        d["taoc"] = float(np.float32(m["tao"].max()))
        d["layer"], d["ql"], d["vel"] = layer, ql, vel
    for k, a in m.items():
        d[k] = np.ascontiguousarray(a, dtype=np.float32)
    return d


def _smooth_noise(g, shape, cells=4.0):
    a = torch.randn(shape, generator=g, device=g.device)
    kx = torch.fft.fftfreq(shape[0], device=g.device)[:, None]
    kz = torch.fft.rfftfreq(shape[1], device=g.device)[None, :]
    a = torch.fft.irfft2(torch.fft.rfft2(a) * torch.exp(-2 * (math.pi * cells) ** 2 * (kx * kx + kz * kz)), s=shape)
    return a / a.std()


def _state(d, seed):
    """A wavefield in full swing: smooth fields in the proportions of a travelling wave."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    amp = (1.0, 2e-7, 2e-7, 2e-3, 2e-3, 4e-10, 4e-10, 5e-2 if d["kind"] in (qpstd.VAPS, qpstd.QRTM) else 0.0)
    return torch.stack([a * _smooth_noise(g, (d["nxx"], d["nzz"])) for a in amp]).cpu().numpy()


def _obs(d, seed):
    """Observed data: a few hyperbolic events of the wavelet on every receiver, already muted."""
    rng = np.random.default_rng(seed)
    t = np.arange(d["nt"])[:, None] * d["dt"]
    off = (np.asarray(d["gxg"]) - d["xsg"])[None, :] * DX
    obs = np.zeros((d["nt"], off.size))
    span = d["nt"] * d["dt"]
    for _ in range(3):
        a = (PI * d["fd"] * (t - np.sqrt((rng.uniform(0.2, 0.9) * span) ** 2 + (off / 9000.0) ** 2))) ** 2
        obs += rng.uniform(-1, 1) * (1 - 2 * a) * np.exp(-a)
    return obs.astype(np.float32)


def _symbol_rows(d, rank):
    """Low-rank factors of the layered window: factor b is the mixed-domain symbol's row of layer b, the last one
    stands for the layers below it too, and ranks above the number of layers add factors without weight."""
    nxx, nzz = d["nxx"], d["nzz"]
    kx = 2 * PI / (nxx * DX) * np.arange(nxx // 2 + 1)
    kz = 2 * PI / (nzz * DX) * np.arange(nzz // 2 + 1)
    k = np.sqrt(kx[:, None] ** 2 + kz[None, :] ** 2)
    k[0, 0] = 1e-6
    U = np.zeros((nxx, nzz, rank), dtype=np.float32)
    V = np.zeros((rank, k.size), dtype=np.float32)
    last = min(rank, len(d["vel"])) - 1
    for b in range(rank):
        vp, q = d["vel"][min(b, last)], d["ql"][min(b, last)]
        gam, tau = 1.0 / PI / q, vp / q
        u = 0.5 * vp * d["dt"] * k ** (1 + gam)
        V[b] = (np.sinc(u / math.pi) * k ** gam * np.sqrt(1 + 0.5 * d["dt"] * tau * k ** 1.01)).ravel()
        if b <= last:
            U[:, np.minimum(d["layer"], last) == b, b] = 1.0
    return {"U": U.reshape(-1, rank), "V": V, "A": np.eye(rank), "nxx": nxx, "nzz": nzz, "row": rank, "col": rank}


def _group(case, seed):
    """The shots of a batch or of a served mix: widths (and for the mix depths and kinds) around the case's."""
    rng = np.random.default_rng(100 * case["nxx"] + case["nzz"])
    out = []
    for i in range(case["shots"]):
        nxx = max(2 * case["pml"] + 30, int(case["nxx"] * rng.uniform(0.5, 1.5)))
        nzz, kind, nt = case["nzz"], case["kind"], case["nt"]
        if case["path"] == "server":
            nzz = max(2 * case["pml"] + 30, int(nzz * rng.uniform(0.5, 1.5)))
            kind = ("aps", "vaps", "artm", "aps", "vaps", "qrtm", "aps", "vaps", "artm", "aps")[i % 10]
            nt = nt * 3 if kind in ("aps", "vaps") else nt
        d = _shot(kind, nxx, nzz, case["pml"], nt, case["dt"], seed * 64 + i, case["snaps"], case["eta"])
        out.append((kind, d, _obs(d, seed * 64 + i + 5) if kind in ("artm", "qrtm") else None))
    return out


def _one(case, seed):
    return _shot(case["kind"], case["nxx"], case["nzz"], case["pml"], case["nt"], case["dt"], seed,
                 case.get("snaps", 0), case.get("eta", 0.0), case.get("rank", 0) > 0)


def prepare(case, seed):
    path = case["path"]
    if path == "steps":
        d = _one(case, seed)
        sh = qpstd.Shot(d)
        if case["rank"]:
            sh.set_lowrank(_symbol_rows(d, case["rank"]))
        sh.set_state(_state(d, seed))
        return dict(path=path, shot=sh, nt=case["nt"])
    if path == "rtm":
        d = _one(case, seed)
        sh = qpstd.Shot(d)
        sh.set_obs(_obs(d, seed + 5))
        return dict(path=path, shot=sh)
    if path == "batch":
        group = _group(case, seed)
        b = qpstd.Batch([d for _, d, _ in group])
        for i, (_, _, obs) in enumerate(group):
            b.set_obs(i, obs)
        return dict(path=path, batch=b, n=len(group))
    if path == "server":
        return dict(path=path, server=qpstd.Server(mem_budget=6 << 30, max_active=16), group=_group(case, seed))
    return dict(path=path, shot=_one(case, seed))


def run(state):
    path = state["path"]
    if path == "steps":
        g = state["shot"].advance(0, state["nt"])
        return [g, list(state["shot"].get_state())]
    if path == "rtm":
        state["shot"].rtm_device()
        return list(state["shot"].get_image())
    if path == "batch":
        state["batch"].rtm_device(8)
        return [list(state["batch"].get_image(i)) for i in range(state["n"])]
    if path == "server":
        sv = state["server"]
        ids = [sv.submit(d, obs) for _, d, obs in state["group"]]
        sv.wait()
        out = []
        for i in ids:
            r = sv.result(i)
            out.append(list(r) if isinstance(r, tuple) else r)
            del sv.keep[i]
        return out
    return qpstd.model_shot(state["shot"])


# ---- what a pass cannot do without ---------------------------------------------------
def _steps_work(kind, nxx, nzz, steps):
    """A step reads and writes the state once and reads the model once (72 bytes a point acoustic, 96
    constant-Q); its transforms are 6 + 6 (acoustic) or 12 + 11 (constant-Q) real line transforms along x and z."""
    n, visco = float(nxx) * nzz, kind in ("vaps", "qrtm")
    lines = (12 * math.log2(nxx) + 11 * math.log2(nzz)) if visco else 6 * (math.log2(nxx) + math.log2(nzz))
    return np.array([(96.0 if visco else 72.0) * n * steps, (2.5 * lines + (70.0 if visco else 40.0)) * n * steps])


def _rtm_steps(nt, snaps):
    """Forward steps of the checkpointed source wavefield plus the receiver steps."""
    reps, rng_ = 0, 1
    while rng_ < nt:
        reps += 1
        rng_ = rng_ * (reps + snaps) // reps
    return reps * nt - rng_ * reps // (snaps + 1) + 2 * nt


def work(case):
    w = np.zeros(2)
    if case["path"] in ("steps", "call"):
        w += _steps_work(case["kind"], case["nxx"], case["nzz"], case["nt"])
    elif case["path"] == "rtm":
        w += _steps_work(case["kind"], case["nxx"], case["nzz"], _rtm_steps(case["nt"], case["snaps"]))
    else:
        for kind, d, obs in _group(case, 0):
            steps = d["nt"] if obs is None else _rtm_steps(d["nt"], d["snaps"])
            w += _steps_work(kind, d["nxx"], d["nzz"], steps)
    return {"bytes": float(w[0]), "flops": float(w[1])}


# ---- the equations in 64 bits ---------------------------------------------------------
class _Exact:
    def __init__(self, d, factors=None):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.d, self.dt = d, float(np.float32(d["dt"]))
        self.visco = d["kind"] in (qpstd.VAPS, qpstd.QRTM)
        nx, nz = d["nxx"], d["nzz"]
        T = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=self.dev)  # noqa: E731
        for k in ("vp", "rho", "bbx", "bbz") + (("gam", "lam", "vwd", "tao") if self.visco else ()):
            setattr(self, k, T(d[k]))
        self.ax, self.bx, self.hax, self.hbx = (T(v)[:, None] for v in self._cpml(nx))
        self.az, self.bz, self.haz, self.hbz = (T(v)[None, :] for v in self._cpml(nz))
        kx, kz = self._k(nx), self._k(nz)
        self.k2 = T(kx)[:, None] ** 2 + T(kz)[None, :] ** 2
        self.ka = self.k2 ** 0.505
        self.dxm, self.dxp = (torch.as_tensor(self._shift(nx, s), device=self.dev)[:, None] for s in (-1, 1))
        self.dzm, self.dzp = (torch.as_tensor(self._shift(nz, s), device=self.dev)[None, :] for s in (-1, 1))
        self.src = np.asarray(d["rik"], dtype=np.float64) * self.dt * 1000.0
        self.gx = torch.as_tensor(np.asarray(d["gxg"]), device=self.dev, dtype=torch.long)
        self.gz = torch.as_tensor(np.asarray(d["gzg"]), device=self.dev, dtype=torch.long)
        self.factors = None
        if factors:
            r, hx, hz = factors["row"], nx // 2 + 1, nz // 2 + 1
            ix, iz = np.minimum(np.arange(nx), nx - np.arange(nx)), np.minimum(np.arange(nz), nz - np.arange(nz))
            V = np.asarray(factors["V"], dtype=np.float64).reshape(r, hx, hz)[:, ix][:, :, iz]
            U = np.asarray(factors["U"], dtype=np.float64) @ factors["A"]
            self.factors = [(T(U[:, b].reshape(nx, nz)), T(V[b])) for b in range(r)]

    def _k(self, n):
        i = np.arange(n)
        return np.where(i < n // 2 + 1, i, n - i) * (2.0 * PI / (n * DX))

    def _shift(self, n, sign):
        """Half-cell shifted derivative along a line of n; the phases mirror about index n/2*2."""
        i = np.arange(n)
        m = np.where(i < n // 2 + 1, i, n // 2 * 2 - i)
        c, s = np.cos(m * PI / n), np.sin(m * PI / n) * np.where(i < n // 2 + 1, 1.0, -1.0)
        a, b = self._k(n) * c, sign * self._k(n) * s
        return np.where(i < n // 2 + 1, -b + 1j * a, b - 1j * a)

    def _cpml(self, n):
        """a, b at the grid points and at the half points."""
        pml, dt = self.d["pml"], self.dt
        amax, dmax = PI * self.d["fd"], 4 * 5000.0 * math.log(1e5) / (2.0 * pml * DX)
        d0, a0, d1, a1 = (np.zeros(n) for _ in range(4))
        i = np.arange(pml)
        d0[:pml], a0[:pml] = dmax * ((pml - 1 - i) / pml) ** 3, amax * i / (pml - 1)
        a0[pml:n - pml] = a0[pml - 1]
        d0[n - pml:], a0[n - pml:] = d0[:pml][::-1], a0[:pml][::-1]
        i = np.arange(pml - 1)
        d1[:pml - 1], a1[:pml - 1] = dmax * ((pml - 1.5 - i) / pml) ** 3, amax * (i + 0.5) / (pml - 1)
        a1[pml - 1:n - pml] = a1[pml - 2]
        d1[n - pml:n - 1], a1[n - pml:n - 1] = d1[:pml - 1][::-1], a1[:pml - 1][::-1]
        a1[n - 1] = a1[n - 2]
        b0, b1 = np.exp(-dt * (d0 + a0)), np.exp(-dt * (d1 + a1))
        return d0 / (d0 + a0) * (b0 - 1), b0, d1 / (d1 + a1) * (b1 - 1), b1

    def _op(self, spec, sym):
        return torch.fft.ifft2(spec * sym).real

    def step(self, s, t, amp=0.0, obs=None, eta=0.0, after_p=None):
        p, vx, vz, fipx, fipz, fivx, fivz, aux = s
        dt = self.dt
        sx = torch.fft.ifft(torch.fft.fft(vx, dim=0) * self.dxm, dim=0).real
        sz = torch.fft.ifft(torch.fft.fft(vz, dim=1) * self.dzm, dim=1).real
        fivx = self.bx * fivx + self.ax * sx
        fivz = self.bz * fivz + self.az * sz
        div = sx + fivx + sz + fivz
        F = torch.fft.fft2(div)
        sg = 1.0 if self.d["kind"] == qpstd.QRTM else -1.0
        if not self.visco:
            p = p + self.rho * self.vp ** 2 * dt * (div - (self.vp * dt) ** 2 / 12.0 * self._op(F, self.k2))
        elif self.factors:
            w = sum(u * self._op(F, v) for u, v in self.factors)
            p = p + self.rho * self.vp ** 2 * dt * w + sg * dt * self.tao * aux
        else:
            tot = (1 - 32 * self.gam) * div + 32 * self.gam * self.vwd * self._op(F, self.k2 ** (1 / 32)) \
                - dt ** 2 * self.vp ** 2 * self.lam / 12.0 * (
                    (1 - 64 * self.gam) * self._op(F, self.k2)
                    + 64 * self.gam * self.vwd * self._op(F, self.k2 ** (33 / 32)))
            D = self._op(torch.fft.fft2(tot), self.ka)
            p = p + self.rho * self.vp ** 2 * dt * self.lam * (tot + sg * 0.5 * dt * self.tao * D) \
                + sg * dt * self.tao * aux
        if amp:
            p[self.d["xsg"], self.d["zsg"]] += amp
        if obs is not None:
            p[self.gx, self.gz] = obs
        if after_p:
            after_p(p)
        gx = torch.fft.ifft(torch.fft.fft(p, dim=0) * self.dxp, dim=0).real
        gz = torch.fft.ifft(torch.fft.fft(p, dim=1) * self.dzp, dim=1).real
        fipx = self.hbx * fipx + self.hax * gx
        fipz = self.hbz * fipz + self.haz * gz
        if self.visco:
            sym = self.ka
            if self.d["kind"] == qpstd.QRTM:
                e6, tao = float(np.float32(eta)) * 1e-6, self.d["taoc"]
                sym = sym - 2 * e6 * sym * (1 + tao * dt * sym) / (
                    torch.exp(-tao * t * dt * sym) + e6 * torch.exp(tao * dt * sym))
            aux = self._op(torch.fft.fft2(p), sym)
        return [p, vx + dt * self.bbx * (gx + fipx), vz + dt * self.bbz * (gz + fipz), fipx, fipz, fivx, fivz, aux]

    def zero(self):
        z = torch.zeros_like(self.vp)
        return [z.clone() for _ in range(8)]

    def model(self, s):
        rows = []
        for t in range(self.d["nt"]):
            s = self.step(s, t, self.src[t], after_p=lambda p: rows.append(p[self.gx, self.gz].clone()))
        return torch.stack(rows), s

    def rtm(self, obs):
        """The source wavelet starts from zero, so a restart from any checkpoint gives the same wavefield and a
        stored history of p stands for the checkpointing."""
        m = self.d["pml"]
        cut = lambda a: a[m:-m, m:-m]  # noqa: E731
        hist, ssg = [], torch.zeros_like(self.vp)
        s = self.zero()
        for t in range(self.d["nt"]):
            s = self.step(s, t, self.src[t], eta=self.d["etas"], after_p=lambda p: hist.append(p.clone()))
        for p in hist:
            ssg += p * p
        img, r = torch.zeros_like(ssg), self.zero()
        rows = torch.as_tensor(np.asarray(obs, dtype=np.float64), device=self.dev)
        for t in range(self.d["nt"] - 1, -1, -1):
            def image(p, t=t):
                img.add_(hist[t] * p)
            r = self.step(r, t, obs=rows[t], eta=self.d["etar"], after_p=image)
        return [cut(img).contiguous(), cut(ssg).contiguous()]


def exact(case, seed):
    path = case["path"]
    if path in ("steps", "call"):
        d = _one(case, seed)
        e = _Exact(d, _symbol_rows(d, case["rank"]) if case["rank"] else None)
        s0 = e.zero() if path == "call" else [torch.as_tensor(a, device=e.dev, dtype=torch.float64)
                                              for a in _state(d, seed)]
        g, s = e.model(s0)
        return g if path == "call" else [g, s]
    if path == "rtm":
        d = _one(case, seed)
        return _Exact(d).rtm(_obs(d, seed + 5))
    out = []
    for kind, d, obs in _group(case, seed):
        e = _Exact(d)
        out.append(e.rtm(obs) if obs is not None else e.model(e.zero())[0])
    return out
