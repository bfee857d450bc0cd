"""Workloads of the library, each as a user's program runs it through tarang_b200's Python API.

A case is a dict of plain values.  ``kind`` says which call it is:

  steps      IncFluid.step(n) and the fields back in host memory: what a simulation does between
             two outputs (the driver loops of the reference run on between outputs in the same way)
  loop       the reference driver's loop body call by call (Compute_force ... Time_advance, energy)
  diag       the output block of a run: energies, shell spectra, fluxes and shell-to-shell tables
  transform  Forward_transform_array / Inverse_transform_array on host arrays
  serve      a batch of independent solves of mixed shapes through serving.Server

``run`` continues from the state that the last pass left, as a simulation does; ``exact`` gives what
the first pass after ``prepare`` returns, from a plain 64-bit torch evaluation of the same equations.
Results of the FP32-mixed form are kept in single precision, its own.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from tarang_b200 import _lib as L
from tarang_b200.serving import Server
from tarang_b200.solver import IncFluid

FORCED = dict(force="supply", inner=2.0, outer=3.0, eps=0.1)
RB = dict(basis="SCFT", physics="RB", Ra=1e6, Pr=1.0, kf=1.0 / math.sqrt(2.0))
NSTATE = {"FLUID": 3, "MHD": 6, "SCALAR": 4, "RB": 4}
ET_KINDS = {"FLUID": (L.TG_ET_UU,), "MHD": (L.TG_ET_UU, L.TG_ET_BB, L.TG_ET_UB, L.TG_ET_BU)}
# the shapes of the serving ensemble: (N1, N2, N3, physics)
SERVED = ((32, 32, 32, "FLUID"), (64, 64, 64, "FLUID"), (128, 128, 128, "FLUID"), (64, 64, 64, "MHD"),
          (65, 128, 128, "RB"))


def _steps(name, N, precision="FP64", n=20, dt=5e-4, nu=1e-3, **kw):
    c = dict(name=name, kind="steps", N1=N[0], N2=N[1], N3=N[2], basis="FOUR", physics="FLUID",
             precision=precision, scheme="RK4", n=n, dt=dt, nu=nu)
    c.update(kw)
    return c


def listed():
    return [
        # forced isotropic turbulence, the headline run, in both arithmetic forms
        _steps("fluid 256 fp64", (256, 256, 256), n=20, **FORCED),
        _steps("fluid 256 mixed", (256, 256, 256), precision="FP32", n=100, **FORCED),
        # decaying MHD turbulence (the largest state: six fields)
        _steps("mhd 256 mixed", (256, 256, 256), physics="MHD", precision="FP32", n=100),
        # Rayleigh-Benard convection, sin/cos basis along the odd axis
        _steps("convection 129x256x256 fp64", (129, 256, 256), n=20, dt=1e-4, **RB),
        _steps("convection 65x128x128 mixed", (65, 128, 128), precision="FP32", n=100, dt=1e-4, **RB),
        # Taylor-Green at 64^3, the small validation run
        _steps("taylor-green 64 fp64", (64, 64, 64), n=100, dt=1e-3, nu=0.01, init="tg"),
        # the smallest solve: a step is a chain of short launches
        _steps("fluid 32 mixed", (32, 32, 32), precision="FP32", n=20, dt=1e-3, nu=5e-3),
        # passive scalar on a box whose x and y lengths are no powers of two
        _steps("scalar 96x80x64 fp64", (96, 80, 64), physics="SCALAR", n=20, dt=1e-3, nu=5e-3),
        # a driver written against the reference: its loop body call by call
        dict(_steps("loop 128 fp64", (128, 128, 128), n=10, nu=3e-3, **FORCED), kind="loop"),
        # the diagnostics a run writes at every output
        dict(_steps("diagnostics mhd 128 fp64", (128, 128, 128), physics="MHD", n=1), kind="diag", shells=16),
        # the bare transforms on host arrays
        dict(name="transform 128 fp64", kind="transform", N1=128, N2=128, N3=128, basis="FOUR", precision="FP64",
             parity=0),
        # request serving: independent solves of the ensemble's shapes, admitted together
        dict(name="serve 20 requests", kind="serve", requests=20, n=20, mix=20261203),
    ]


def _len(rng, lo, hi, pow2):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if rng.random() < pow2:
        return 1 << max(4, min(8, int(round(math.log2(v)))))
    return 2 * int(round(v / 2))


def draw(rng):
    kind = rng.choice(("steps",) * 6 + ("loop", "diag", "transform", "serve"))
    if kind == "serve":
        return dict(kind="serve", requests=rng.randint(4, 20), n=rng.randint(4, 20), mix=rng.randint(1, 10**6))
    physics = rng.choice(("FLUID", "FLUID", "MHD", "SCALAR", "RB"))
    if kind == "diag":
        physics = rng.choice(("FLUID", "MHD"))
    N3 = 1 << rng.randint(5, 8)
    hi = 256 if kind in ("steps", "transform") else 160
    N1, N2 = _len(rng, 32, hi, 0.6), _len(rng, 32, hi, 0.6)
    if kind in ("loop", "diag"):
        N3 = min(N3, 128)
    basis = "FOUR"
    if physics == "RB":
        basis, N1 = "SCFT", max(17, min(129, N1 // 2 + rng.randint(0, 1)))
    if kind == "transform":
        if rng.random() < 0.3:
            basis, N1 = "SCFT", min(129, N1 + 1)
        return dict(kind="transform", N1=min(N1, 160), N2=min(N2, 160), N3=min(N3, 128), basis=basis,
                    precision=rng.choice(("FP64", "FP32")), parity=rng.randint(0, 1))
    odd = sum(1 for v in (N1, N2) if v & (v - 1)) if basis == "FOUR" else (1 if N2 & (N2 - 1) else 0)
    cost = N1 * N2 * N3 * NSTATE[physics] / 3.0 * (1 + 3 * odd)
    n = max(2, min(100, int(rng.uniform(0.3, 1.0) * 10 * 256**3 / cost)))
    c = dict(kind=kind, N1=N1, N2=N2, N3=N3, basis=basis, physics=physics,
             precision=rng.choice(("FP64", "FP32")), scheme=rng.choice(("RK4",) * 6 + ("RK2", "EULER")),
             n=min(n, 10) if kind == "loop" else n, dt=round(rng.uniform(2e-4, 1e-3), 6),
             nu=round(math.exp(rng.uniform(math.log(3e-3), math.log(1e-2))), 5))
    if physics == "RB":
        c.update(Ra=10 ** rng.randint(4, 6), Pr=rng.choice((0.7, 1.0, 6.8)), kf=1.0 / math.sqrt(2.0), dt=1e-4)
    elif physics in ("FLUID", "MHD") and rng.random() < 0.5:
        c.update(FORCED)
    if kind == "diag":
        c.update(n=1, shells=rng.randint(8, 20), precision="FP64", scheme="RK4")
    return c


# ------------------------------------------------------------------ inputs
def _grid(c):
    """Wavenumbers (broadcastable), |K|^2 and the stored (2/3) modes of a case's spectral grid."""
    N1, N2, N3 = c["N1"], c["N2"], c["N3"]
    dev = "cuda"
    kf = (c.get("kf"), c.get("kf")) if c.get("kf") else (1.0, 1.0)
    l1, l2, l3 = (torch.arange(n, device=dev, dtype=torch.float64) for n in (N1, N2, N3 // 2 + 1))
    if c["basis"] == "FOUR":
        ix = torch.where(l1 <= N1 // 2, l1, l1 - N1)
        keep_x = ix.abs() < N1 // 3
    else:
        ix, keep_x = l1, l1 < 2 * N1 // 3
    iy = torch.where(l2 <= N2 // 2, l2, l2 - N2)
    keep_y = (l2 < N2 // 3) | (l2 > 2 * N2 // 3 + 1)
    keep_z = l3 < N3 // 3
    fx = math.pi if c["basis"] == "SCFT" else 1.0
    f2 = math.pi * kf[0] if c["basis"] == "SCFT" else kf[0]
    kx, ky, kz = (ix * fx)[:, None, None], (iy * f2)[None, :, None], (l3 * f2)[None, None, :]
    keep = keep_x[:, None, None] & keep_y[None, :, None] & keep_z[None, None, :]
    return kx, ky, kz, kx * kx + ky * ky + kz * kz, keep


def _kfactor(c):
    return (math.pi, math.pi * c["kf"], math.pi * c["kf"]) if c["basis"] == "SCFT" else (1.0, 1.0, 1.0)


def _weights(c):
    """Energy weight of a mode: 1/2 on kz = 0 else 1 (FOUR); doubled for kx > 0 (SCFT); 0 at the origin."""
    w = torch.ones((c["N1"], c["N2"], c["N3"] // 2 + 1), dtype=torch.float64, device="cuda")
    w[:, :, 0] = 0.5
    if c["basis"] == "SCFT":
        w[1:] *= 2.0
    w[0, 0, 0] = 0.0
    return w


def _dx(c, a, sine):
    """x derivative of a coefficient array (a sine series if `sine`, of no account in FOUR)."""
    kx = c["_grid"][0]
    if c["basis"] == "FOUR":
        return 1j * kx * a
    return kx * a if sine else -kx * a


def _project(c, v):
    """Divergence-free part of three component arrays."""
    _, ky, kz, K2, _ = c["_grid"]
    inv = torch.where(K2 > 0, 1.0 / K2.clamp(min=1e-300), torch.zeros_like(K2))
    p = inv * (_dx(c, v[0], True) + 1j * (ky * v[1] + kz * v[2]))
    return [v[0] + _dx(c, p, False), v[1] + 1j * ky * p, v[2] + 1j * kz * p]


def _noise(c, gen, peak, slope, sine=False):
    """Coefficients of a real random field, amplitude ~ k^slope exp(-(k / peak)^2)."""
    shape = (c["N1"], c["N2"], c["N3"])
    r = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    a = torch.fft.rfftn(r, dim=(0, 1, 2) if c["basis"] == "FOUR" else (1, 2), norm="forward")
    _, _, _, K2, keep = c["_grid"]
    a = a * torch.where(keep, K2 ** (slope / 2) * torch.exp(-K2 / peak**2), torch.zeros_like(K2))
    a[0, 0, 0] = 0
    if sine:
        a[0] = 0
    return a


def _scaled(c, v, energy):
    e = sum((_weights(c) * a.abs() ** 2).sum() for a in v)
    return [a * torch.sqrt(energy / e) for a in v]


def _initial(case, seed):
    """State fields of a case on the device, complex128, reference layout."""
    c = dict(case)
    c["_grid"] = _grid(c)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    phys = c["physics"]
    if c.get("init") == "tg":
        # the Taylor-Green vortex with a small random disturbance
        N = (c["N1"], c["N2"], c["N3"])
        x, y, z = (torch.arange(n, device="cuda", dtype=torch.float64) * (2 * math.pi / n) for n in N)
        x, y, z = x[:, None, None], y[None, :, None], z[None, None, :]
        r = [torch.sin(x) * torch.cos(y) * torch.cos(z), -torch.cos(x) * torch.sin(y) * torch.cos(z),
             torch.zeros(N, device="cuda", dtype=torch.float64)]
        base = [torch.fft.rfftn(a, norm="forward") for a in r]
        d = _scaled(c, _project(c, [_noise(c, gen, 4.0, 1.0) for _ in range(3)]), 1e-3)
        return [a + b for a, b in zip(base, d)], c
    if phys == "RB":
        v = [_noise(c, gen, 16.0, 0.0, sine=(i == 0)) for i in range(3)]
        v = _scaled(c, _project(c, v), 1e-2)
        v[0][0] = 0
        return v + _scaled(c, [_noise(c, gen, 16.0, 0.0, sine=True)], 1e-2), c
    peak = 4.0  # E(k) ~ k^4 exp(-2 (k/4)^2)
    v = _scaled(c, _project(c, [_noise(c, gen, peak, 1.0) for _ in range(3)]), 0.5)
    if phys == "MHD":
        v += _scaled(c, _project(c, [_noise(c, gen, peak, 1.0) for _ in range(3)]), 0.5)
    elif phys == "SCALAR":
        v += _scaled(c, [_noise(c, gen, peak, 1.0)], 0.5)
    return v, c


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True)


def _config(c):
    kw = dict(N=(c["N1"], c["N2"], c["N3"]), basis=c["basis"], physics=c["physics"], precision=c["precision"],
              nu=c["nu"], dt=c["dt"], scheme=c["scheme"], kfactor=_kfactor(c), n_shells=c.get("shells", 12))
    if c.get("force") == "supply":
        kw["force"] = dict(inner=c["inner"], outer=c["outer"], eps=c["eps"])
    if c["physics"] == "RB":
        kw.update(Ra=c["Ra"], Pr=c["Pr"])
    return kw


def _field_ids(physics):
    ids = [L.TG_V1, L.TG_V2, L.TG_V3]
    if physics == "MHD":
        ids += [L.TG_W1, L.TG_W2, L.TG_W3]
    elif physics in ("SCALAR", "RB"):
        ids += [L.TG_T]
    return ids


def _requests(case):
    """The requests of a serving case: plain step cases, FP32-mixed, one viscosity each."""
    rs = np.random.RandomState(case["mix"])
    out = []
    for _ in range(case["requests"]):
        N1, N2, N3, phys = SERVED[rs.randint(len(SERVED))]
        nu = float(np.exp(rs.uniform(math.log(1e-3), math.log(1e-2))))
        N = (N1, N2, N3)
        if phys == "RB":
            out.append(_steps("", N, precision="FP32", n=case["n"], nu=nu, dt=1e-4, **RB))
        else:
            out.append(_steps("", N, physics=phys, precision="FP32", n=case["n"], nu=nu))
    return out


def prepare(case, seed):
    if case["kind"] == "serve":
        reqs = _requests(case)
        fields = []
        for i, r in enumerate(reqs):
            v, _ = _initial(r, seed * 1000 + i)
            h = _pinned((len(v), r["N1"], r["N2"], r["N3"] // 2 + 1), torch.complex128)
            for k, a in enumerate(v):
                h[k].copy_(a)
            fields.append(h.numpy())
        srv = Server(hbm_budget=16e9, max_batch=32, borrow_inputs=True)
        return dict(case=case, srv=srv, cfg=[_config(r) for r in reqs], fields=fields)
    if case["kind"] == "transform":
        N = (case["N1"], case["N2"], case["N3"])
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        # real data in the packed layout: N3 reals and two of padding in a row
        r = torch.zeros((N[0], N[1], N[2] + 2), dtype=torch.float64, device="cuda")
        r[:, :, : N[2]] = torch.randn(N, generator=gen, device="cuda", dtype=torch.float64)
        real = torch.view_as_complex(r.reshape(N[0], N[1], N[2] // 2 + 1, 2)).cpu().numpy()
        kw = dict(basis="SCFT", physics="RB", Ra=1e6, Pr=1.0) if case["basis"] == "SCFT" else {}
        U = IncFluid(N, precision=case["precision"], **kw)
        return dict(case=case, U=U, real=real)
    v, c = _initial(case, seed)
    U = IncFluid(**_config(case))
    shape = (case["N1"], case["N2"], case["N3"] // 2 + 1)
    host = [_pinned(shape, torch.complex128) for _ in v]
    for i, (f, a) in enumerate(zip(_field_ids(case["physics"]), v)):
        host[i].copy_(a)
        U.upload(f, host[i].numpy())
        # the driver's arrays hold the stored modes; the rest is zero
        host[i].copy_(torch.where(c["_grid"][4], a, torch.zeros_like(a)))
    s = dict(case=case, U=U, host=host, ids=_field_ids(case["physics"]))
    if case["precision"] == "FP32":
        s["single"] = [torch.zeros(shape, dtype=torch.complex64) for _ in v]
    return s


def _fields(s):
    for f, h in zip(s["ids"], s["host"]):
        s["U"].download_stored(f, h.numpy())
    if s["case"]["precision"] != "FP32":
        return [h.numpy() for h in s["host"]]
    for d, h in zip(s["single"], s["host"]):
        torch.view_as_real(d).copy_(torch.view_as_real(h))
    return s["single"]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "serve":
        srv = s["srv"]
        ids = [srv.submit(cfg, f, case["n"]) for cfg, f in zip(s["cfg"], s["fields"])]
        srv.drain()
        out = []
        for i in ids:
            out.append(torch.from_numpy(srv.result(i)[0].base).to(torch.complex64))
            srv.release(i)
        return out
    U = s["U"]
    if kind == "transform":
        spec = U.Forward_transform_array(s["real"], case["parity"])
        back = U.Inverse_transform_array(spec, case["parity"])
        if case["precision"] == "FP32":
            return [torch.from_numpy(a).to(torch.complex64) for a in (spec, back)]
        return [spec, back]
    if kind == "steps":
        e = U.step(case["n"])
        return dict(energy=e if case["precision"] != "FP32" else e.astype(np.float32), fields=_fields(s))
    if kind == "loop":
        es = []
        for _ in range(case["n"]):
            U.Compute_force()
            U.Compute_nlin()
            U.Add_force()
            U.Compute_pressure()
            U.Get_dt()
            U.Time_advance()
            es.append(U.CV_Compute_totalenergy_diss()[0])
        return dict(energy=np.array(es, dtype=np.float64 if case["precision"] != "FP32" else np.float32),
                    fields=_fields(s))
    out = dict(flux=[], transfer=[], spectrum=[])
    groups = (0, 1) if case["physics"] == "MHD" else (0,)
    out["energy"] = [list(U.CV_Compute_totalenergy_diss(g)) for g in groups]
    for g in groups:
        out["spectrum"] += list(U.CV_Compute_shell_spectrum(g))
    for k in ET_KINDS[case["physics"]]:
        out["flux"].append(U.Compute_flux(k))
        out["transfer"].append(U.Compute_shell_tr(k))
    return out


# ------------------------------------------------------------------ bytes and operations
def _work_step(c):
    """One RK step.  A three-dimensional transform of fields larger than the chip takes two passes
    over memory (x; y and z): every transformed field crosses it once in between, on the stored ky
    and kz.  Transformed: the state fields, and the products of a stage (the pressure takes the
    trace of u_i u_j, so 5 for a fluid, 8 with a scalar or a magnetic field)."""
    N1, N2, N3 = c["N1"], c["N2"], c["N3"]
    t = 8 if c["precision"] == "FP32" else 16
    ns = NSTATE[c["physics"]]
    nt = ns + (5 if ns == 3 else 8)
    stages = {"RK4": 4, "RK2": 2, "EULER": 1}[c["scheme"]]
    nky, nkz = 2 * N2 / 3.0, N3 / 3.0
    nkx = 2 * N1 / 3.0
    stage = nt * 2 * N1 * nky * nkz * t
    state = 2 * ns * nkx * nky * nkz * 16
    points = N1 * N2 * N3
    return stages * stage + state, stages * nt * 2.5 * points * math.log2(points)


def work(case):
    if case["kind"] == "serve":
        w = [_work_step(r) for r in _requests(case)]
        return dict(bytes=case["n"] * sum(b for b, _ in w), flops=case["n"] * sum(f for _, f in w))
    points = case["N1"] * case["N2"] * case["N3"]
    if case["kind"] == "transform":
        # each transform reads its array and writes it, twice (x; y and z)
        return dict(bytes=2 * 2 * 2 * 8.0 * points, flops=2 * 2.5 * points * math.log2(points))
    if case["kind"] == "diag":
        # per giver shell and kind: 3 inverse and 9 forward transforms
        n = len(ET_KINDS[case["physics"]]) * (case["shells"] - 1)
        stored = points / 4.5
        return dict(bytes=n * 12 * 2 * stored * 16, flops=n * 12 * 2.5 * points * math.log2(points))
    b, f = _work_step(case)
    return dict(bytes=case["n"] * b, flops=case["n"] * f)


# ------------------------------------------------------------------ the same in 64 bits
class _Plain:
    """The equations of a case in plain torch, 64 bits, on the dense grid."""

    def __init__(self, c):
        self.c = c
        self.N = (c["N1"], c["N2"], c["N3"])
        self.kx, self.ky, self.kz, self.K2, self.keep = c["_grid"]
        if c["basis"] == "SCFT":
            n, m = self.N[0], torch.arange(self.N[0], device="cuda", dtype=torch.float64)
            th = math.pi * m[:, None] * (2 * m[None, :] + 1) / (2 * n)  # [mode][point]
            self.cosm, self.sinm = torch.cos(th), torch.sin(th)
        d = 3
        kf = _kfactor(c)
        nx = self.N[0] // d if c["basis"] == "FOUR" else 2 * self.N[0] // 3
        self.kin = int(min(nx * kf[0], (self.N[1] // d) * kf[1], (self.N[2] // d) * kf[2]))
        self.kout = int(math.ceil(math.sqrt((nx * kf[0]) ** 2 + ((self.N[1] // d) * kf[1]) ** 2
                                            + ((self.N[2] // d) * kf[2]) ** 2)))
        self.w = _weights(c)
        phys = c["physics"]
        nu = c["nu"]
        self.nu = [nu] * NSTATE[phys]
        if phys == "RB":
            self.nu = [math.sqrt(c["Pr"] / c["Ra"])] * 3 + [1.0 / math.sqrt(c["Ra"] * c["Pr"])]
        if c.get("force") == "supply":
            k = torch.sqrt(self.K2)
            self.band = torch.nonzero((k > c["inner"]) & (k <= c["outer"]), as_tuple=True)
            cnt = 0
            r = int(math.ceil(c["outer"]))
            for i in range(-r, r + 1):
                for j in range(-r, r + 1):
                    for q in range(r + 1):
                        if c["inner"] <= math.sqrt(i * i + j * j + q * q) < c["outer"]:
                            cnt += 1 if q == 0 else 2
            self.e_mode = c["eps"] / cnt

    def inv(self, a, sine=False):
        N1, N2, N3 = self.N
        if self.c["basis"] == "FOUR":
            return torch.fft.irfftn(a, s=self.N, norm="forward")
        r = torch.fft.irfftn(a, s=(N2, N3), dim=(1, 2), norm="forward").reshape(N1, -1)
        if sine:
            return (2 * self.sinm.T @ r).reshape(self.N)
        s = r.clone()
        s[1:] *= 2
        return (self.cosm.T @ s).reshape(self.N)

    def fwd(self, r, sine=False):
        N1, N2, N3 = self.N
        if self.c["basis"] == "FOUR":
            return torch.fft.rfftn(r, norm="forward")
        m = (self.sinm if sine else self.cosm) @ r.reshape(N1, -1)
        return torch.fft.rfftn(m.reshape(self.N), dim=(1, 2), norm="forward") / N1

    def d(self, a, j, sine=False):
        return _dx(self.c, a, sine) if j == 0 else 1j * (self.ky if j == 1 else self.kz) * a

    def advect(self, f, sf, u, su):
        """D_j F(u_j f_i); sf, su: whether f_i, u_j are sine series along x."""
        out = []
        for i in range(len(f)):
            t = 0
            for j in range(3):
                s = sf[i] != su[j]
                t = t + self.d(self.fwd(u[j] * f[i], s), j, s)
            out.append(torch.where(self.keep, t, torch.zeros_like(t)))
        return out

    def supply(self, v):
        """alpha V + beta omega on the band, at a given energy and no helicity per mode."""
        at = self.band
        x = [a[at] for a in v]
        k = [t.expand(self.K2.shape)[at] for t in (self.kx, self.ky, self.kz)]
        km = torch.sqrt(self.K2[at])
        E = 0.5 * sum(a.abs() ** 2 for a in x)
        cr = [x[1].real * x[2].imag - x[2].real * x[1].imag, x[2].real * x[0].imag - x[0].real * x[2].imag,
              x[0].real * x[1].imag - x[1].real * x[0].imag]
        s = (k[0] * cr[0] + k[1] * cr[1] + k[2] * cr[2]) / (km * E)
        al = self.e_mode / (2 * E) / (1 - s * s)
        be = -al * s
        be = torch.where(be > 1e-15, be, torch.zeros_like(be))
        om = [1j * (k[1] * x[2] - k[2] * x[1]), 1j * (k[2] * x[0] - k[0] * x[2]), 1j * (k[0] * x[1] - k[1] * x[0])]
        return [al * a + be * o for a, o in zip(x, om)]

    def rhs(self, f):
        c = self.c
        scft = c["basis"] == "SCFT"
        par = [scft, False, False]
        u = [self.inv(a, p) for a, p in zip(f[:3], par)]
        if c["physics"] == "MHD":
            b = [self.inv(a) for a in f[3:]]
            n = [x - y for x, y in zip(self.advect(u, par, u, par), self.advect(b, par, b, par))]
            nb = [x - y for x, y in zip(self.advect(b, par, u, par), self.advect(u, par, b, par))]
        else:
            n, nb = self.advect(u, par, u, par), []
            if len(f) > 3:
                nb = self.advect([self.inv(f[3], scft)], [scft], u, par)
        if c["physics"] == "RB":
            n[0] = n[0] - f[3]
            nb[0] = nb[0] - f[0]
        if c.get("force") == "supply":
            for a, g in zip(n, self.supply(f[:3])):
                a[self.band] -= g
        return [-a for a in _project(c, n)] + [-a for a in nb]

    def energy(self, f, n=None):
        n = n or (6 if self.c["physics"] == "MHD" else 3)
        return sum(float((self.w * a.abs() ** 2).sum()) for a in f[:n])

    def step(self, f):
        c = self.c
        E0 = self.energy(f)
        dt = min(2 * math.pi / max(1, self.kin) / (math.sqrt(E0) * 20), c["dt"]) if E0 > 0 else c["dt"]
        two = [torch.exp(-nu * 0.5 * dt * self.K2) for nu in sorted(set(self.nu))]
        at = [sorted(set(self.nu)).index(nu) for nu in self.nu]
        h = [two[i] for i in at]
        r = self.rhs(f)
        if c["scheme"] == "EULER":
            return [e * e * (a + dt * x) for e, a, x in zip(h, f, r)]
        u = [e * (a + dt / 2 * x) for e, a, x in zip(h, f, r)]
        if c["scheme"] == "RK2":
            r = self.rhs(u)
            return [e * (e * a + dt * x) for e, a, x in zip(h, f, r)]
        tot = [dt / 6 * e * e * x for e, x in zip(h, r)]
        r = self.rhs(u)
        u = [e * a + dt / 2 * x for e, a, x in zip(h, f, r)]
        tot = [t + dt / 3 * e * x for t, e, x in zip(tot, h, r)]
        r = self.rhs(u)
        u = [e * (e * a + dt * x) for e, a, x in zip(h, f, r)]
        tot = [t + dt / 3 * e * x for t, e, x in zip(tot, h, r)]
        r = self.rhs(u)
        return [e * e * a + t + dt / 6 * x for e, a, t, x in zip(h, f, tot, r)]

    def run(self, f, n):
        es = []
        f = [torch.where(self.keep, a, torch.zeros_like(a)) for a in f]
        for _ in range(n):
            f = self.step(f)
            # a step's energy is U's and B's, the driver's loop asks for U's
            es.append(self.energy(f, 3 if self.c["kind"] == "loop" else None))
        return np.array(es), f

    # diagnostics (FOUR)
    def spectrum(self, v):
        K = torch.sqrt(self.K2)
        b = torch.ceil(K).long()
        n = self.kout + 1
        mult = torch.ones_like(self.K2)
        mult[:, :, 0] = 0.5
        nyq = torch.zeros(self.K2.shape, dtype=torch.bool, device="cuda")
        nyq[self.N[0] // 2] = True
        nyq[:, self.N[1] // 2] = True
        mult = torch.where(nyq, 2 * mult, mult)
        sel = b < n

        def bins(x):
            return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, b[sel], x[sel])

        cnt = bins(mult)
        r = torch.arange(n, device="cuda", dtype=torch.float64)
        f = torch.where((r > self.kin) & (cnt >= 1), 2 * math.pi * r * r / cnt.clamp(min=1), torch.ones_like(r))
        ek = torch.stack([bins(mult * a.abs() ** 2) * f for a in v])
        dk = 2 * sum(bins(mult * self.K2 * a.abs() ** 2) * f for a in v)
        return ek, dk

    def transfers(self, kind, U, B):
        S = self.c["shells"]
        rin = float(self.kin)
        R = [0.0, 2.0, 4.0, 8.0] + [0.0] * (S - 3)
        for i in range(4, S - 2):
            R[i] = 8 * 2.0 ** (math.log2(rin / 16.0) / (S - 5) * (i - 3))
        R[S - 2], R[S - 1], R[S] = rin / 2, rin, 1e4
        H, F, G, sign = {L.TG_ET_UU: (U, U, U, -1), L.TG_ET_BB: (U, B, B, -1), L.TG_ET_UB: (B, U, B, 1),
                         L.TG_ET_BU: (U, B, U, 1)}[kind]
        K = torch.sqrt(self.K2)
        m2 = 2 * self.w
        m2[0, 0, 0] = 1.0
        h = [self.inv(a) for a in H]
        idx = torch.full(K.shape, S + 1, device="cuda", dtype=torch.long)
        for i in range(S, -1, -1):
            idx = torch.where(K <= R[i], i, idx)

        def density(lo, hi):
            g = [self.inv(torch.where((K > lo) & (K <= hi), a, torch.zeros_like(a))) for a in F]
            n = self.advect(g, [False] * 3, h, [False] * 3)
            return m2 * sum((x * y.conj()).real for x, y in zip(n, G))

        flux = torch.zeros(S + 1, dtype=torch.float64, device="cuda")
        tr = torch.zeros((S + 1, S + 1), dtype=torch.float64, device="cuda")
        for s in range(1, S + 1):
            d = density(0.0, R[s])
            flux[s] = sign * d[(K > R[s]) & (K <= 1e4)].sum()
        inside = K <= rin
        for s in range(1, S):
            d = density(R[s - 1], R[s])
            tr[s] = sign * torch.zeros(S + 2, dtype=torch.float64, device="cuda").index_add_(
                0, idx[inside], d[inside])[: S + 1]
        return flux, tr


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":
        out = []
        for i, r in enumerate(_requests(case)):
            v, c = _initial(r, seed * 1000 + i)
            out.append(torch.stack(_Plain(c).run(v, case["n"])[1]))
        return out
    if kind == "transform":
        N = (case["N1"], case["N2"], case["N3"])
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        real = torch.randn(N, generator=gen, device="cuda", dtype=torch.float64)
        c = dict(case, physics="FLUID", nu=0.0, kf=1.0)
        c["_grid"] = _grid(c)
        p = _Plain(c)
        spec = p.fwd(real, case["parity"] == 1)
        back = torch.zeros((N[0], N[1], N[2] + 2), dtype=torch.float64, device="cuda")
        back[:, :, : N[2]] = p.inv(spec, case["parity"] == 1)
        return [spec, torch.view_as_complex(back.reshape(N[0], N[1], N[2] // 2 + 1, 2))]
    v, c = _initial(case, seed)
    p = _Plain(c)
    if kind in ("steps", "loop"):
        points = case["N1"] * case["N2"] * case["N3"]
        if points * case["n"] > 2.2e9:
            return None
        e, f = p.run(v, case["n"])
        return dict(energy=e, fields=f)
    v = [torch.where(p.keep, a, torch.zeros_like(a)) for a in v]
    U, B = v[:3], v[3:]
    out = dict(flux=[], transfer=[], spectrum=[], energy=[])
    for g in ([U, B] if B else [U]):
        out["energy"].append([float(sum((p.w * a.abs() ** 2).sum() for a in g)),
                              float(2 * sum((p.w * p.K2 * a.abs() ** 2).sum() for a in g))])
        out["spectrum"] += list(p.spectrum(g))
    for k in ET_KINDS[case["physics"]]:
        f, t = p.transfers(k, U, B)
        out["flux"].append(f)
        out["transfer"].append(t)
    return out
