"""The work that users of the engine give it, as timed cases.

Each case is one pass through the public entry points, with the inputs that a
program holds before the call already in hand:

  model      seismograms of a batch of shots: Engine.forward (host arrays) or
             Engine.forward_device (CUDA tensors)
  objective  an FWI line-search objective: new model, modelling on the device,
             misfit reduction (as inversion.fwi.objective_function)
  gradient   an FWI iteration's gradient: new model, exact gradient and source
             illumination (as inversion.fwi.calculate_gradient)
  migrate    reverse-time migration of a batch with the mute armed, and the
             normalised image (as migration.SolveBackwardWaveEquation)
  refgrad    the reference-form gradient, with the anisotropy parameters'
             gradients for VTI and TTI

Grids, spacings, time steps, wavelets, borders and acquisition follow
workloads.py and the tests; runs are shortened in time on the large grids so
that a pass stays below a second.  exact() evaluates the same schemes in 64-bit
torch.
"""
import math

import numpy as np
import torch

from pseudoacousticmodeling_gb300 import Config, Engine
from pseudoacousticmodeling_gb300.engine import BOUNDARY_SAVING


def _case(name, kind, approx, boundary, nz, nx, border, shots, samples, **more):
    c = dict(kind=kind, approx=approx, boundary=boundary, nz=nz, nx=nx, border=border, shots=shots, samples=samples,
             h=10.0, dt=0.001, fcut=15.0, rec_every=1, spread=False, device=False, every=0, store="f32")
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one shot of the small two-layer model at full length, through host arrays: the reference user's first run
        _case("shot_acoustic", "model", "acoustic", "cerjan", 201, 401, 50, 1, 2001),
        # one shot with the perfectly matched layer on a ragged grid
        _case("shot_acoustic_cpml", "model", "acoustic", "CPML", 287, 653, 45, 1, 1201),
        # one anisotropic shot with the reference's own border: a quick look at a field-size VTI model
        _case("shot_vti", "model", "VTI", "cerjan", 401, 1001, 50, 1, 801, fcut=12.0, dt=0.0008),
        # the batched VTI survey with the matched layer, sources and seismograms resident on the GPU
        _case("batch_vti_cpml", "model", "VTI", "CPML", 801, 2001, 50, 64, 301, fcut=12.0, dt=0.0008, device=True),
        # a batched TTI survey with the reference's border
        _case("batch_tti", "model", "TTI", "cerjan", 601, 1501, 50, 16, 301, h=8.0, dt=0.0006, fcut=12.0, device=True),
        # a line-search objective of acoustic FWI over the whole survey
        _case("objective_acoustic", "objective", "acoustic", "cerjan", 501, 1701, 50, 64, 401, fcut=8.0, device=True),
        # its gradient: checkpoints in HBM, the source field recomputed in segments
        _case("gradient_acoustic", "gradient", "acoustic", "cerjan", 501, 1701, 50, 32, 401, fcut=8.0, every=300),
        # the gradient of one shot at a time, every step stored, on a small model
        _case("gradient_shot", "gradient", "acoustic", "cerjan", 201, 401, 50, 1, 1201),
        # acoustic migration, split-spread receivers, half-precision checkpoints
        _case("migrate_acoustic", "migrate", "acoustic", "cerjan", 501, 2001, 50, 8, 801, h=5.0, dt=0.0004, fcut=30.0,
              spread=True, rec_every=2, every=200, store="f16"),
        # acoustic migration of two shots with the matched layer and boundary saving, ragged sizes
        _case("migrate_cpml_bands", "migrate", "acoustic", "CPML", 259, 611, 40, 2, 901, every=BOUNDARY_SAVING),
        # VTI migration on the modelling grid, checkpoints
        _case("migrate_vti", "migrate", "VTI", "cerjan", 801, 2001, 50, 8, 201, fcut=12.0, dt=0.0008, every=200),
        # multiparameter TTI gradient of a few shots on a ragged grid
        _case("refgrad_tti", "refgrad", "TTI", "cerjan", 251, 601, 40, 4, 501, dt=0.0008),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model", "model", "model", "objective", "gradient", "migrate", "migrate", "refgrad"])
    nz, nx = _logint(rng, 60, 800), _logint(rng, 90, 2000)
    border = rng.choice([20, 30, 35, 40, 45, 50, 50, 60])
    shots = _logint(rng, 1, 64)
    approx = rng.choice(["acoustic", "VTI", "TTI"])
    boundary = "cerjan"
    if approx != "TTI" and kind == "model":
        boundary = rng.choice(["cerjan", "CPML"])
    every, store = 0, "f32"
    if kind in ("objective", "gradient"):
        approx = "acoustic"
    if kind == "migrate":
        if approx == "acoustic":
            boundary = rng.choice(["cerjan", "CPML"])
        every = rng.choice([0, 100, 200, BOUNDARY_SAVING])
        store = rng.choice(["f32", "f32", "bf16", "f16"])
    if kind == "gradient":
        every = rng.choice([0, 200, 300])
    h, dt, fcut = rng.choice([(10.0, 0.001, 15.0), (10.0, 0.0008, 12.0), (8.0, 0.0006, 15.0), (10.0, 0.001, 12.0)])
    cells = (nz + 2 * border) * (nx + 2 * border)
    # cell updates of a pass, and the bytes that storing every step takes, within those of the listed cases
    cap = {"model": 2.5e10, "objective": 2.5e10, "gradient": 1.2e10, "migrate": 6e9, "refgrad": 1.2e9}[kind]
    lag = int(round(2.0 * math.sqrt(math.pi) / fcut / dt))
    shots = max(1, min(shots, int(cap / (cells * (lag + 150)))))
    most = min(1500, max(150, int(cap / (cells * shots)) - lag))
    samples = rng.randint(101, max(most, 120))
    if every == 0 and kind in ("gradient", "migrate", "refgrad"):
        shots = max(1, min(shots, int(2.0e10 / (4.0 * cells * (lag + samples)))))
    return _case(None, kind, approx, boundary, nz, nx, border, shots, samples, h=h, dt=dt, fcut=fcut,
                 rec_every=rng.choice([1, 2, 3]), spread=rng.random() < 0.3,
                 device=kind == "objective" or (kind == "model" and rng.random() < 0.5), every=every, store=store)


# ------------------------------------------------------------------ inputs

def _lag(c):
    return int(round(2.0 * math.sqrt(math.pi) / c["fcut"] / c["dt"]))


def _smooth(g, nz, nx, lo, hi):
    """A smooth random field: coarse noise, bicubic in between."""
    f = torch.rand(1, 1, max(nz // 25, 2) + 3, max(nx // 25, 2) + 3, generator=g)
    f = torch.nn.functional.interpolate(f, size=(nz, nx), mode="bicubic", align_corners=False)[0, 0].clamp(0.0, 1.0)
    return (lo + (hi - lo) * f).numpy()


def _inputs(c, seed):
    """Models, wavelet, geometry and observed data of a case, from the seed alone."""
    g = torch.Generator().manual_seed(seed)
    rng = np.random.default_rng(seed)
    nz, nx, N, B, h = c["nz"], c["nx"], c["border"], c["shots"], c["h"]
    lag, nt = _lag(c), _lag(c) + c["samples"]
    depths = np.sort(rng.uniform(0.1, 0.9, 4))
    layer = np.searchsorted(depths * (nz - 1), np.arange(nz))
    vp = np.float32(1500.0 + 500.0 * layer)[:, None] + _smooth(g, nz, nx, 0.0, 250.0)
    q = {"vp": np.ascontiguousarray(vp, np.float32), "eps": None, "delta": None, "theta": None}
    if c["approx"] != "acoustic":
        q["eps"] = _smooth(g, nz, nx, 0.0, 0.25)
        q["delta"] = _smooth(g, nz, nx, 0.0, 0.1)
    if c["approx"] == "TTI":
        q["theta"] = _smooth(g, nz, nx, -40.0, 40.0)
    t = np.arange(nt) * c["dt"] - 2.0 * math.sqrt(math.pi) / c["fcut"]
    fc = c["fcut"] / (3.0 * math.sqrt(math.pi))
    arg = math.pi ** 3 * fc * fc * t * t
    q["wavelet"] = ((1.0 - 2.0 * arg) * np.exp(-arg) / (h * h)).astype(np.float32)
    first = rng.integers(0, max(nx // 8, 1))
    q["sx"] = (N + np.linspace(first, nx - 1, B).round()).astype(np.int32)
    q["sz"] = np.full(B, N + 1, np.int32)
    cols = np.arange(0, nx, c["rec_every"])
    if c["spread"]:
        # a spread of its own for each shot, half the line long and centred on the source where the line allows
        n = max(cols.size // 2, 1)
        lo = np.clip((q["sx"] - N) // c["rec_every"] - n // 2, 0, cols.size - n)
        q["rx"] = (N + cols[lo[:, None] + np.arange(n)]).astype(np.int32)
    else:
        q["rx"] = (N + cols).astype(np.int32)
    q["rz"] = np.full_like(q["rx"], N + 2)
    if c["kind"] in ("model",):
        return q
    # observed data: a direct wave, two reflections and a little noise per gather
    rx = np.broadcast_to(q["rx"], (B, q["rx"].shape[-1]))
    x = torch.from_numpy(((rx - q["sx"][:, None]) * h).astype(np.float32)).cuda()
    d = torch.zeros(B, c["samples"], x.shape[-1], device="cuda")
    tt = (torch.arange(c["samples"], device="cuda") * c["dt"])[None, :, None]
    for t0, v, amp in zip((0.0, rng.uniform(0.15, 0.3), rng.uniform(0.3, 0.6)), (1550.0, 1900.0, 2300.0), (1.0, 0.3, 0.2)):
        a = math.pi ** 3 * fc * fc * (tt - torch.sqrt(t0 * t0 + (x / v) ** 2)[:, None, :]) ** 2
        d += amp * (1.0 - 2.0 * a) * torch.exp(-a)
    d += 0.01 * torch.randn(d.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))
    q["dobs"] = d.mul_(1.0 / (h * h))
    return q


def prepare(case, seed):
    c = dict(case)
    q = _inputs(c, seed)
    nt = _lag(c) + c["samples"]
    e = Engine(Config(nz=c["nz"], nx=c["nx"], n_abc=c["border"], dz=c["h"], dx=c["h"], dt=c["dt"], nt=nt,
                      itlag=_lag(c), fcut=c["fcut"], approximation=c["approx"], boundary=c["boundary"],
                      max_shots=c["shots"]))
    e.set_wavelet(q["wavelet"])
    e.set_receivers(q["rz"], q["rx"], per_shot=c["spread"])
    s = {"c": c, "q": q, "e": e}
    if c["kind"] in ("model", "migrate", "refgrad"):
        e.set_models(q["vp"], q["eps"], q["delta"], q["theta"])
    if c["kind"] == "refgrad" and c["approx"] != "acoustic":
        e.set_multiparameter(True)
    if c["device"]:
        s["stream"] = torch.cuda.Stream()
        s["d_sz"], s["d_sx"] = torch.from_numpy(q["sz"]).cuda(), torch.from_numpy(q["sx"]).cuda()
        s["seis"] = torch.empty(c["shots"], c["samples"], q["rx"].shape[-1], device="cuda")
    elif "dobs" in q:
        pinned = torch.empty(q["dobs"].shape, dtype=torch.float32, pin_memory=c["kind"] == "gradient")
        pinned.copy_(q.pop("dobs"))
        s["keep"] = pinned
        q["dobs"] = pinned.numpy()
    return s


def run(s):
    c, q, e = s["c"], s["q"], s["e"]
    kind = c["kind"]
    if kind == "model":
        if c["device"]:
            e.forward_device(s["d_sz"], s["d_sx"], s["seis"], stream=s["stream"].cuda_stream)
            return s["seis"]
        return e.forward(q["sz"], q["sx"])
    if kind == "objective":
        e.set_models(q["vp"])
        e.forward_device(s["d_sz"], s["d_sx"], s["seis"], stream=s["stream"].cuda_stream)
        return s["seis"], e.misfit_device(s["seis"], q["dobs"], stream=s["stream"].cuda_stream)
    if kind == "gradient":
        e.set_models(q["vp"])
        e.rtm_reset()
        misfit, grad = e.misfit_gradient(q["sz"], q["sx"], q["dobs"], ckpt_interval=c["every"], store=c["store"])
        return misfit, grad, e.fwi_result()[1]
    if kind == "migrate":
        e.rtm_reset()
        h = c["h"]
        e.set_mute((q["sx"] - c["border"]) * h, (q["sz"] - c["border"]) * h, (q["rx"] - c["border"]) * h,
                   (q["rz"] - c["border"]) * h, 1500.0, 0.1, 0.05)
        e.rtm(q["sz"], q["sx"], q["dobs"], ckpt_interval=c["every"], store=c["store"])
        return e.rtm_result(norm="py")
    e.rtm_reset()
    misfit = e.fwi_gradient(q["sz"], q["sx"], q["dobs"], ckpt_interval=c["every"], store=c["store"])
    out = [misfit, *e.fwi_result()]
    if c["approx"] != "acoustic":
        out += [v for v in e.fwi_multiparameter_result() if v is not None]
    return out


def work(case):
    """One time step of one shot reads two fields and writes one (12 B a cell);
    the backward step of a migration or gradient does so for the receiver field
    and reads the source field once more.  The models are read once a step for
    the batch.  Seismograms and images are small beside that."""
    c = case
    B, N = c["shots"], c["border"]
    nz, nx = c["nz"] + 2 * N, c["nx"] + 2 * N
    nt = _lag(c) + c["samples"]
    models = {"acoustic": 1, "VTI": 3, "TTI": 4}[c["approx"]]
    flops = {"acoustic": 33, "VTI": 75, "TTI": 104}[c["approx"]]
    strips = 0
    if c["boundary"] == "CPML":          # psi and zeta of the strip cells, read and written
        strips = 2 * N * (nz + nx) * 16
    step = B * (12 * nz * nx + strips) + 4 * models * nz * nx
    data = 4 * B * c["samples"] * len(range(0, c["nx"], c["rec_every"])) // (2 if c["spread"] else 1)
    if c["kind"] in ("model", "objective"):
        return {"bytes": nt * step + data * (1 if c["kind"] == "model" else 3), "flops": nt * B * nz * nx * flops}
    back = step + 4 * B * nz * nx
    if c["every"] > 0:                   # the segments before the last are modelled again
        again = (nt - 1) // c["every"] * c["every"]
    else:
        again = nt if c["every"] < 0 else 0
    more = {"acoustic": 4, "VTI": 100, "TTI": 150}[c["approx"]]
    return {"bytes": (nt + again) * step + nt * back + data,
            "flops": (2 * nt + again) * B * nz * nx * flops + nt * B * nz * nx * more}


# ------------------------------------------------------------------ 64-bit evaluation

C8 = (-1435.0 / 504.0, 8.0 / 5.0, -1.0 / 5.0, 8.0 / 315.0, -1.0 / 560.0)
A8 = (0.0, 4.0 / 5.0, -1.0 / 5.0, 4.0 / 105.0, -1.0 / 280.0)


def _sh(U, k, axis):
    """U shifted by k cells along an axis, the four outer cells of it cut off."""
    n = U.shape[axis] - 8
    return U.narrow(axis, 4 + k, n)


def _cut(U, axis):
    return U.narrow(axis, 4, U.shape[axis] - 8)


def _d2(U, axis, inv):
    """Second derivative, on the cells that have four neighbours on both sides along the axis."""
    out = _sh(U, 0, axis) * (C8[0] * inv * inv)
    for k in range(1, 5):
        out.add_(_sh(U, k, axis), alpha=C8[k] * inv * inv).add_(_sh(U, -k, axis), alpha=C8[k] * inv * inv)
    return out


def _d1(U, axis, inv):
    out = _sh(U, 1, axis) * (A8[1] * inv)
    out.sub_(_sh(U, -1, axis), alpha=A8[1] * inv)
    for k in range(2, 5):
        out.add_(_sh(U, k, axis), alpha=A8[k] * inv).sub_(_sh(U, -k, axis), alpha=A8[k] * inv)
    return out


class _Scheme:
    """The scheme of one case in 64 bits for some of its shots."""

    def __init__(self, c, q):
        N, h = c["border"], c["h"]
        self.c, self.q, self.N, self.inv = c, q, N, 1.0 / h
        self.dt = float(np.float32(c["dt"]))
        pad = lambda a: torch.from_numpy(np.pad(a, N, mode="edge").astype(np.float64)).cuda()  # noqa: E731
        vp = pad(q["vp"])
        self.vp, self.nz, self.nx = vp, *vp.shape
        self.kap = (vp * vp * self.dt * self.dt)[4:-4, 4:-4]
        if c["approx"] != "acoustic":
            self.eps, self.delta = pad(q["eps"])[4:-4, 4:-4], pad(q["delta"])[4:-4, 4:-4]
            th = torch.deg2rad(pad(q["theta"]))[4:-4, 4:-4] if c["approx"] == "TTI" else torch.zeros_like(self.eps)
            self.cos, self.sin = torch.cos(th), torch.sin(th)
        self.D = torch.ones(self.nz, self.nx, dtype=torch.float64, device="cuda")
        if c["boundary"] == "cerjan":
            i = torch.arange(N, dtype=torch.float64, device="cuda")
            a = torch.exp(-((N - i) / (1.4142 * 3.0 * N)) ** 2)
            self.D[:, :N] *= a
            self.D[:, -N:] *= a.flip(0)
            self.D[:N] *= a[:, None]
            self.D[-N:] *= a.flip(0)[:, None]
        self.D = self.D[4:-4, 4:-4].contiguous()

    def zeros(self, B):
        return torch.zeros(B, self.nz, self.nx, dtype=torch.float64, device="cuda")

    def strips(self, B):
        """Zero memory variables: [axis][side] of (psi, zeta), strips along the last axis of U or of its transpose."""
        W, z = self.N - 4, torch.float64
        n = {2: self.nz - 8, 1: self.nx - 8}
        return {ax: [[torch.zeros(B, n[ax], W, dtype=z, device="cuda") for _ in range(2)] for _ in range(2)] for ax in (2, 1)}

    def profile(self, axis):
        """(a, b) of the strips on both sides along an axis, shaped like the strips."""
        c, N, h = self.c, self.N, self.c["h"]
        v = self.vp if axis == 2 else self.vp.T
        n = v.shape[1]
        d0 = -3.0 * math.log(1e-3 ** (N / 10.0))
        out = []
        for side, i in enumerate((torch.arange(4, N), torch.arange(n - N, n - 4))):
            r = ((N - i - 1.0) if side == 0 else (i - n + N)).double().cuda() / N
            d = d0 / (2.0 * N * h) * r * r * v[4:-4, i.cuda()]
            al = math.pi * c["fcut"] / 3.0 * (1.0 - r * r)
            a = torch.exp(-(d + al) * self.dt)
            out.append((a, torch.where((d + al).abs() > 1e-10, d / (d + al) * (a - 1.0), 0.0)))
        return out

    def advance_strips(self, U, mem, ab):
        """Memory variables of U's step; returns the terms added to (dx, dz, dxx, dzz) as [axis][side]."""
        terms = {}
        for axis in (2, 1):
            V = U if axis == 2 else U.transpose(1, 2)
            V = V[:, 4:-4]
            n, N = V.shape[2], self.N
            terms[axis] = []
            for side in (0, 1):
                w = V[:, :, :N + 4] if side == 0 else V[:, :, n - N - 4:]
                a, b = ab[axis][side]
                psi, zeta = mem[axis][side]
                psi.mul_(a).add_(b * _d1(w, 2, self.inv))
                dpsi = _d1(torch.nn.functional.pad(psi, (4, 4)), 2, self.inv)
                # the strip next to the other cells: its neighbours' psi is zero
                zeta.mul_(a).add_(b * (_d2(w, 2, self.inv) + dpsi))
                terms[axis].append((dpsi, dpsi + zeta))
        return terms

    def add_strips(self, terms, dx, dz, dxx, dzz):
        W = self.N - 4
        for axis, d1, d2 in ((2, dx, dxx), (1, dz, dzz)):
            for side in (0, 1):
                g, h = terms[axis][side]
                if axis == 1:
                    g, h = g.transpose(1, 2), h.transpose(1, 2)
                at = slice(0, W) if side == 0 else slice(-W, None)
                s = (slice(None), slice(None), at) if axis == 2 else (slice(None), at, slice(None))
                if d1 is not None:
                    d1[s] += g
                d2[s] += h

    def operator(self, U, terms=None):
        """kappa times the spatial operator of U, on the update region."""
        approx, inv = self.c["approx"], self.inv
        Ux, Uz = _cut(U, 1), _cut(U, 2)
        dxx, dzz = _d2(Ux, 2, inv), _d2(Uz, 1, inv)
        if approx == "acoustic":
            if terms:
                self.add_strips(terms, None, None, dxx, dzz)
            return dxx.add_(dzz).mul_(self.kap)
        dx, dz = _d1(Ux, 2, inv), _d1(Uz, 1, inv)
        if terms:
            self.add_strips(terms, dx, dz, dxx, dzz)
        e2, ct, st = 1.0 + 2.0 * self.eps, self.cos, self.sin
        if approx == "TTI":
            dx, dz = dx * ct - dz * st, dx * st + dz * ct
        x2, z2 = dx.square_(), dz.square_()
        den = e2 * x2 * x2 + z2 * z2 + 2.0 * (1.0 + self.delta) * x2 * z2
        sd = torch.where(den.abs() > 1e-12, -2.0 * (self.eps - self.delta) * x2 * z2 / den, 0.0)
        if approx == "VTI":
            return dxx.mul_(e2 + sd).add_(dzz.mul_(1.0 + sd)).mul_(self.kap)
        out = dxx.mul_(e2 * ct * ct + st * st + sd).add_(dzz.mul_(e2 * st * st + ct * ct + sd))
        out.sub_(_d1(_d1(U, 1, inv), 2, inv).mul_(4.0 * self.eps * st * ct))
        return out.mul_(self.kap)

    def source_fields(self, shots, record, keep):
        """Runs the shots forward.  Returns the seismograms (if asked) and the
        damped fields U(t) of every step after its update (if asked)."""
        c, q = self.c, self.q
        B, nt, lag = len(shots), _lag(c) + c["samples"], _lag(c)
        b = torch.arange(B, device="cuda")
        sz, sx = (torch.from_numpy(q[k][shots].astype(np.int64)).cuda() for k in ("sz", "sx"))
        rz, rx, rb = self.receivers(shots)
        w = torch.from_numpy(q["wavelet"].astype(np.float64)).cuda()
        cur, nxt = self.zeros(B), self.zeros(B)
        cpml = c["boundary"] == "CPML"
        mem, ab = (self.strips(B), {ax: self.profile(ax) for ax in (2, 1)}) if cpml else (None, None)
        seis = torch.zeros(B, c["samples"], rx.shape[-1], dtype=torch.float64, device="cuda") if record else None
        kept, raw = [], []
        for k in range(nt):
            cur[b, sz, sx] += w[k]
            if keep == "raw":
                raw.append(cur.clone())
            terms = self.advance_strips(cur, mem, ab) if cpml else None
            inner, old = cur[:, 4:-4, 4:-4], nxt[:, 4:-4, 4:-4]
            old.neg_().add_(inner, alpha=2.0).add_(self.operator(cur, terms))
            old.mul_(self.D)
            inner.mul_(self.D)
            if record and k >= lag:
                seis[:, k - lag] = cur[rb, rz, rx]
            if keep == "damped":
                kept.append(cur.clone())
            cur, nxt = nxt, cur
        return seis, raw if keep == "raw" else kept

    def receivers(self, shots):
        q, B = self.q, len(shots)
        rz, rx = (np.broadcast_to(a[shots] if a.ndim == 2 else a, (B, a.shape[-1])).astype(np.int64) for a in (q["rz"], q["rx"]))
        rb = torch.arange(B, device="cuda")[:, None].expand(B, rx.shape[-1])
        return torch.from_numpy(rz.copy()).cuda(), torch.from_numpy(rx.copy()).cuda(), rb

    def anisotropic_adjoint(self, U, P):
        """kappa times the adjoint operator on the receiver field U with the source field P."""
        inv, e, d = self.inv, self.eps, self.delta
        Px, Pz = _cut(P, 1), _cut(P, 2)
        lap = _d2(Px, 2, inv).add_(_d2(Pz, 1, inv))
        dx, dz = _d1(Px, 2, inv), _d1(Pz, 1, inv)
        ct, st, e2 = self.cos, self.sin, 1.0 + 2.0 * e
        xr, zr = dx * ct - dz * st, dx * st + dz * ct
        x2, z2 = xr * xr, zr * zr
        den = e2 * x2 * x2 + z2 * z2 + 2.0 * (1.0 + d) * x2 * z2
        on = den.abs() > 1e-12
        safe = torch.where(on, den, 1.0)
        sd = torch.where(on, -2.0 * (e - d) * x2 * z2 / safe, 0.0)
        f = torch.where(on, 4.0 * (e - d) * xr * zr * (e2 * x2 * x2 - z2 * z2) / (safe * safe), 0.0)
        inner = U[:, 4:-4, 4:-4]
        pad = lambda v: torch.nn.functional.pad(v, (4, 4, 4, 4))  # noqa: E731
        out = _d2(_cut(pad((e2 * ct * ct + st * st + sd) * inner), 1), 2, inv)
        out.add_(_d2(_cut(pad((e2 * st * st + ct * ct + sd) * inner), 2), 1, inv))
        out.sub_(_d1(_cut(pad(lap * f * dz * inner), 1), 2, inv))
        out.add_(_d1(_cut(pad(lap * f * dx * inner), 2), 1, inv))
        if self.c["approx"] == "TTI":
            out.sub_(_d1(_d1(pad(4.0 * e * st * ct * inner), 1, inv), 2, inv))
        return out.mul_(self.kap)

    def backward(self, shots, P, data, start, stop, each):
        """The receiver field from step `start` down to `stop`, driven by data [B][samples][nrec];
        calls each(t, field) after the injection of step t."""
        c, lag = self.c, _lag(self.c)
        B = len(shots)
        rz, rx, rb = self.receivers(shots)
        cur, nxt = self.zeros(B), self.zeros(B)
        cpml = c["boundary"] == "CPML"
        mem, ab = (self.strips(B), {ax: self.profile(ax) for ax in (2, 1)}) if cpml else (None, None)
        for t in range(start, stop - 1, -1):
            if t >= lag:
                cur.index_put_((rb, rz, rx), data[:, t - lag] * (self.inv * self.inv), accumulate=True)
            each(t, cur)
            if c["approx"] == "acoustic":
                op = self.operator(cur, self.advance_strips(cur, mem, ab) if cpml else None)
            else:
                op = self.anisotropic_adjoint(cur, P[t])
            inner, old = cur[:, 4:-4, 4:-4], nxt[:, 4:-4, 4:-4]
            old.neg_().add_(inner, alpha=2.0).add_(op).mul_(self.D)
            inner.mul_(self.D)
            cur, nxt = nxt, cur

    def parameter_terms(self, P, adj):
        """Sums over the shots of the epsilon, delta and theta gradient terms of one step, on the interior."""
        N, inv = self.N, self.inv
        U = P[:, N:-N, N:-N]
        inn = slice(N, self.nz - 8 - N)      # interior cells with four neighbours inside, in the models' update region
        e, d, ct, st = (m[inn, N:self.nx - 8 - N] for m in (self.eps, self.delta, self.cos, self.sin))
        Ux, Uz = _cut(U, 1), _cut(U, 2)
        pxx, pzz, px, pz = _d2(Ux, 2, inv), _d2(Uz, 1, inv), _d1(Ux, 2, inv), _d1(Uz, 1, inv)
        tti = self.c["approx"] == "TTI"
        pxz = _d1(_d1(U, 1, inv), 2, inv) if tti else torch.zeros_like(pxx)
        h, g = px * ct - pz * st, px * st + pz * ct
        m = torch.maximum(h.abs(), g.abs())
        on = m > 0
        m = torch.where(on, m, 1.0)
        h, g = h / m, g / m
        t = h * h * g * g
        num, den = -2.0 * (e - d) * t, (1.0 + 2.0 * e) * h ** 4 + g ** 4 + 2.0 * (1.0 + d) * t
        den2 = torch.where(on, den * den, 1.0)
        dse = torch.where(on, (-2.0 * t * den - num * 2.0 * h ** 4) / den2, 0.0)
        dsd = torch.where(on, (2.0 * t * den - num * 2.0 * t) / den2, 0.0)
        A = adj[:, 4:-4, 4:-4]
        s2 = 2.0 * st * ct
        ge = A * (-(2.0 * ct * ct + dse) * pxx - (2.0 * st * st + dse) * pzz + 2.0 * s2 * pxz)
        out = [ge.sum(0), (A * (-dsd * (pxx + pzz))).sum(0)]
        if tti:
            w = -2.0 * h * g ** 3 + 2.0 * h ** 3 * g
            dn = -2.0 * (e - d) * w
            dd = -4.0 * (1.0 + 2.0 * e) * h ** 3 * g + 4.0 * h * g ** 3 + 2.0 * (1.0 + d) * w
            dst = torch.where(on, (dn * den - num * dd) / den2, 0.0)
            c2 = ct * ct - st * st
            out.append((A * ((2.0 * e * s2 - dst) * pxx + (-2.0 * e * s2 - dst) * pzz + 4.0 * e * c2 * pxz)).sum(0))
        return out


def _muted(c, q):
    d = torch.from_numpy(q["dobs"]).double().cuda()
    h, N, dt = c["h"], c["border"], float(np.float32(c["dt"]))
    rx, rz = (torch.from_numpy(np.broadcast_to(a, (c["shots"], a.shape[-1])).copy()).cuda() for a in (q["rx"], q["rz"]))
    sx, sz = (torch.from_numpy(a).cuda()[:, None] for a in (q["sx"], q["sz"]))
    t1 = torch.sqrt(((rx - sx) * h).double() ** 2 + ((rz - sz) * h).double() ** 2) / 1500.0 + 0.1
    t = (torch.arange(c["samples"], device="cuda") * dt)[None, :, None].double()
    return d * ((t - t1[:, None]) / 0.05).clamp(0.0, 1.0)


def exact(case, seed):
    c = dict(case)
    q = _inputs(c, seed)
    if "dobs" in q:
        q["dobs"] = q["dobs"].cpu().numpy()
    S = _Scheme(c, q)
    N, B, nt = c["border"], c["shots"], _lag(c) + c["samples"]
    field = S.nz * S.nx * 8.0
    updates = B * S.nz * S.nx * float(nt)
    # seconds of the evaluation, from the passes over memory of one cell update
    passes = {"acoustic": 60, "VTI": 140, "TTI": 200}[c["approx"]]
    back = {"model": 0.0, "objective": 0.0, "gradient": 1.2, "migrate": 1.2, "refgrad": 2.0}[c["kind"]]
    if updates * 8.0 * passes * (1.0 + back) / 4e12 + nt * 1e-3 > 20.0:
        return None
    inner = (slice(None), slice(N, -N), slice(N, -N))
    if c["kind"] in ("model", "objective"):
        step = max(1, int(2e9 / field))
        seis = torch.cat([S.source_fields(np.arange(a, min(a + step, B)), True, None)[0] for a in range(0, B, step)])
        if c["kind"] == "model":
            return seis
        return seis, 0.5 * float((seis - torch.from_numpy(q["dobs"]).cuda()).square().sum())
    step = max(1, int(4e10 / (field * nt)))
    z = lambda n: torch.zeros(c["nz"], c["nx"], dtype=torch.float64, device="cuda") if n else None  # noqa: E731
    img, ilum, misfit = z(1), z(1), 0.0
    gk = torch.zeros(S.nz, S.nx, dtype=torch.float64, device="cuda")
    par = [z(1)[4:-4, 4:-4] for _ in range(3)]
    data = _muted(c, q) if c["kind"] == "migrate" else torch.from_numpy(q["dobs"]).double().cuda()
    for a in range(0, B, step):
        shots = np.arange(a, min(a + step, B))
        d = data[a:a + len(shots)]
        if c["kind"] == "migrate":
            _, P = S.source_fields(shots, False, "damped")

            def each(t, U):
                img.add_((U[inner] * P[t][inner]).sum(0))
                ilum.add_(P[t][inner].square().sum(0))
            S.backward(shots, P, d, nt - 1, 0, each)
            continue
        seis, P = S.source_fields(shots, True, "raw" if c["kind"] == "gradient" else "damped")
        r = seis - d
        misfit += 0.5 * float(r.square().sum())
        for p in P:
            ilum.add_(p[inner].square().sum(0))
        if c["kind"] == "refgrad":
            def each(t, U):
                d2 = (P[t + 1][inner] - 2.0 * P[t][inner] + P[t - 1][inner]) / (S.dt * S.dt)
                img.add_((U[inner] * d2).sum(0))
                if c["approx"] != "acoustic":
                    for total, v in zip(par, S.parameter_terms(P[t], U[inner])):
                        total.add_(v)
            S.backward(shots, P, -r, nt - 2, 1, each)
            continue
        # the exact adjoint on w = kappa D lambda: w(t) = D (2 w(t+1) - D w(t+2) + kappa L w(t+1)) + kappa D^2 r(t)
        rz, rx, rb = S.receivers(shots)
        full = torch.nn.functional.pad(S.kap * S.D * S.D, (4, 4, 4, 4))
        cur, nxt, lag = S.zeros(len(shots)), S.zeros(len(shots)), _lag(c)
        inv = S.inv
        for t in range(nt - 1, -1, -1):
            if t <= nt - 2:
                lap = _d2(_cut(P[t], 1), 2, inv).add_(_d2(_cut(P[t], 2), 1, inv))
                gk[4:-4, 4:-4].add_((cur[:, 4:-4, 4:-4] * lap).sum(0))
            w1, w2 = cur[:, 4:-4, 4:-4], nxt[:, 4:-4, 4:-4]
            w2.mul_(S.D).neg_().add_(w1, alpha=2.0).add_(S.operator(cur)).mul_(S.D)
            if t >= lag:
                nxt.index_put_((rb, rz, rx), r[:, t - lag] * full[rz, rx], accumulate=True)
            cur, nxt = nxt, cur
    if c["kind"] == "migrate":
        return img / (ilum + 1e-5 * ilum.max()), ilum
    if c["kind"] == "refgrad":
        out = [misfit, img, ilum]
        if c["approx"] != "acoustic":
            out += [torch.nn.functional.pad(v, (4, 4, 4, 4)) for v in par[:3 if c["approx"] == "TTI" else 2]]
        return out
    # fold the edge-replicated padding back onto the model, then d kappa / d vp = 2 vp dt^2 on G = kappa dJ/dkappa
    zi = (torch.arange(S.nz, device="cuda") - N).clamp(0, c["nz"] - 1)
    xi = (torch.arange(S.nx, device="cuda") - N).clamp(0, c["nx"] - 1)
    rows = torch.zeros(c["nz"], S.nx, dtype=torch.float64, device="cuda").index_add_(0, zi, gk)
    img.index_add_(1, xi, rows)
    return misfit, img * 2.0 / S.vp[N:-N, N:-N], ilum
