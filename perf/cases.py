"""Performance cases: what a program built on ghost_b200 spends its GPU time on.

Every case goes through the public entry points (`Ghost`, `Ensemble`, `MLP`,
`LES`) the way a solver's time loop, output step or training loop calls them.
Inputs are developed-looking fields: random phases under a k^-5/3 spectrum,
solenoidal, partly helical, inside the 2/3 truncation, <|v|^2> = 1.

A case is a dict of plain values; `kind` selects the path:
  hd     steps of the HD solver (hd_run)
  bouss  steps of the rotating stratified Boussinesq solver (bouss_run)
  mhd    steps of the MHD solver (mhd_run)
  ens    steps of an ensemble of uneven HD runs (Ensemble.run)
  fft    one real-to-complex and one complex-to-real 3D transform
  diag   an output step: global quantities, spectra, transfer function
  train  MLP training steps, then the weights
  infer  MLP inference
  les    steps of an LES run with one of its closures (LES.run)
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ghost_b200 import GHOST_COMPLEX_TO_REAL, GHOST_REAL_TO_COMPLEX, Ensemble, Ghost
from ghost_b200.les import LES, MLP, NHID, NIN, NOUT

DEV = "cuda"


# --------------------------------------------------------------------- cases
def _hd(nx, ny, nz, prec, ord, forced, steps=1):
    return dict(kind="hd", nx=nx, ny=ny, nz=nz, prec=prec, ord=ord, forced=forced, steps=steps)


def listed():
    return [
        # the smallest production grid (64^3 FP64 decay, RK2): ten launches, latency counts
        dict(_hd(64, 64, 64, "fp64", 2, False), name="hd_64_f64"),
        # an everyday double-precision forced run
        dict(_hd(256, 256, 256, "fp64", 4, True), name="hd_256_f64_forced"),
        # the headline: forced turbulence at 512^3 in single precision, RK4
        dict(_hd(512, 512, 512, "fp32", 4, True), name="hd_512_f32_forced"),
        # the largest: rotating stratified flow on an elongated box, RK4
        dict(kind="bouss", nx=1024, ny=1024, nz=256, Lz=0.25, prec="fp32", ord=4, forced=False, steps=1,
             name="bouss_1024x1024x256_f32"),
        # a double-precision MHD run
        dict(kind="mhd", nx=128, ny=128, nz=128, prec="fp64", ord=2, forced=True, steps=1, name="mhd_128_f64"),
        # 256 independent runs of three sizes advanced together
        dict(kind="ens", n0=32, r0=128, n1=64, r1=96, n2=128, r2=32, prec="fp32", ord=2, steps=1, name="ens_256_runs_f32"),
        # transforms called by a host code one field at a time: a large cubic grid ...
        dict(kind="fft", nx=512, ny=512, nz=512, prec="fp32", name="fft_512_f32"),
        # ... and a small non-cubic one
        dict(kind="fft", nx=256, ny=128, nz=64, prec="fp64", name="fft_256x128x64_f64"),
        # the output step of a large run: hdcheck, maxabs, spectra, transfer function
        dict(kind="diag", nx=512, ny=512, nz=512, prec="fp32", name="diag_512_f32"),
        # training the subgrid closure: eight minibatches, forward, backward, Adam
        dict(kind="train", batch=65536, steps=8, name="mlp_train_65536"),
        # the learned closure in a 128^3 LES (inputs, inference, stress divergence, RK4 substeps)
        dict(kind="les", n=128, kc=42, closure="mlp", prec="fp32", ord=4, steps=1, name="les_128_mlp"),
        # GHOST's eddy-viscosity closure in a small LES: launch-bound
        dict(kind="les", n=64, kc=21, closure="edqnm", prec="fp32", ord=4, steps=1, name="les_64_edqnm"),
    ]


def _grid(rng, lo, hi):
    """Three powers of two in 16..1024 with lo <= log2(product) <= hi."""
    while True:
        e = [rng.randint(4, 10) for _ in range(3)]
        t = rng.uniform(lo, hi)
        if abs(sum(e) - t) < 1.0 and max(e) - min(e) <= 4:
            return [1 << q for q in e]


def draw(rng):
    kind = rng.choice(["hd", "hd", "fft", "fft", "bouss", "mhd", "diag", "train", "infer", "les", "ens"])
    prec = rng.choice(["fp32", "fp64"])
    wide = 26 if prec == "fp32" else 25
    if kind == "hd":
        nx, ny, nz = _grid(rng, 12, wide)
        return _hd(nx, ny, nz, prec, rng.choice([2, 3, 4]), rng.random() < 0.6)
    if kind == "fft":
        nx, ny, nz = _grid(rng, 12, wide)
        return dict(kind="fft", nx=nx, ny=ny, nz=nz, prec=prec)
    if kind == "diag":
        nx, ny, nz = _grid(rng, 15, wide)
        return dict(kind="diag", nx=nx, ny=ny, nz=nz, prec=prec)
    if kind == "bouss":
        nx, ny, nz = _grid(rng, 14, wide - 1)
        return dict(kind="bouss", nx=nx, ny=ny, nz=nz, Lz=rng.choice([0.25, 0.5, 1.0]), prec=prec,
                    ord=rng.choice([2, 4]), forced=rng.random() < 0.5, steps=1)
    if kind == "mhd":
        nx, ny, nz = _grid(rng, 14, wide - 2)
        return dict(kind="mhd", nx=nx, ny=ny, nz=nz, prec=prec, ord=2, forced=rng.random() < 0.5, steps=1)
    if kind == "train":
        return dict(kind="train", batch=int(round(math.exp(rng.uniform(math.log(100), math.log(262144))))),
                    steps=rng.choice([1, 4, 8]))
    if kind == "infer":
        return dict(kind="infer", batch=int(round(math.exp(rng.uniform(math.log(50), math.log(2200000))))))
    if kind == "les":
        n = rng.choice([32, 64, 128])
        return dict(kind="les", n=n, kc=n // 3, closure=rng.choice(["none", "edqnm", "mlp", "mlp_spectral"]),
                    prec=prec, ord=rng.choice([2, 4]), steps=1)
    n0, n1, n2 = sorted(rng.sample([16, 32, 64, 128], 3))
    return dict(kind="ens", n0=n0, r0=rng.randint(1, 64), n1=n1, r1=rng.randint(1, 32), n2=n2, r2=rng.randint(1, 12),
                prec=prec, ord=2, steps=1)


# -------------------------------------------------------------------- inputs
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _rdtype(prec):
    return torch.float32 if prec == "fp32" else torch.float64


class _K:
    """Wavenumbers of a grid as broadcastable tensors over (nx/2+1, ny, nz)."""

    def __init__(self, nx, ny, nz, dtype, Lz=None):
        self.n = (nx, ny, nz)
        self.N = float(nx * ny * nz)
        fi = lambda n: torch.cat([torch.arange(0, n // 2), torch.arange(-n // 2, 0)]).to(DEV, dtype)  # noqa: E731
        ix = fi(nx)[:nx // 2 + 1].view(-1, 1, 1)
        iy, iz = fi(ny).view(1, -1, 1), fi(nz).view(1, 1, -1)
        self.Dkk = 1.0
        self.k = [ix, iy, iz]
        if Lz is not None:
            self.k = [ix, iy, iz / Lz]
            self.Dkk = min(1.0, 1.0 / Lz)
        self.kk2 = self.k[0] ** 2 + self.k[1] ** 2 + self.k[2] ** 2
        if Lz is not None or not nx == ny == nz:
            kn2 = ix ** 2 / nx ** 2 + iy ** 2 / ny ** 2 + iz ** 2 / nz ** 2
            kmax = 1.0 / 9.0
        else:
            kn2, kmax = self.kk2, nx * nx / 9.0
        self.kn2 = kn2
        nmax = int(max(nx, ny, nz / (Lz or 1.0)) / self.Dkk)
        self.nbins = nmax // 2 + 1
        self.mask = (kn2 <= kmax) & (kn2 >= min(1e-5, 0.1 / nmax ** 2))
        self.w = torch.full((nx // 2 + 1, 1, 1), 2.0, dtype=dtype, device=DEV)
        self.w[0] = 1.0


def _spectrum(K, gen, dtype, runs, lo, hi, slope):
    """A random-phase spectrum (runs, nx/2+1, ny, nz) of a real field."""
    nx, ny, nz = K.n
    r = torch.randn((runs, nz, ny, nx), dtype=dtype, device=DEV, generator=gen)
    a = torch.fft.rfftn(r, dim=(1, 2, 3)).permute(0, 3, 2, 1)
    del r
    kk = K.kk2.sqrt()
    amp = torch.where(K.mask & (kk >= lo) & (kk <= hi), kk.clamp(min=0.5) ** slope, torch.zeros_like(kk))
    return (a * amp).contiguous()


def _solenoidal(K, gen, dtype, runs=1, lo=0.5, hi=1e9, slope=-11.0 / 6.0, power=1.0):
    """Three fields of a solenoidal, partly helical velocity with <|v|^2> = power."""
    u = [_spectrum(K, gen, dtype, runs, lo, hi, slope) for _ in range(3)]
    k2 = torch.where(K.kk2 > 0, K.kk2, torch.ones_like(K.kk2))
    s = (K.k[0] * u[0] + K.k[1] * u[1] + K.k[2] * u[2]) / k2
    for q in range(3):
        u[q] -= K.k[q] * s
    del s
    ik = 0.5j / k2.sqrt()
    v = [u[q] + ik * (K.k[(q + 1) % 3] * u[(q + 2) % 3] - K.k[(q + 2) % 3] * u[(q + 1) % 3]) for q in range(3)]
    del u
    e = sum((K.w * (x.real ** 2 + x.imag ** 2)).sum(dim=(1, 2, 3), dtype=torch.float64) for x in v) / K.N ** 2
    c = (power / e).sqrt().to(dtype).view(-1, 1, 1, 1)
    return [(x * c).contiguous() for x in v]


def _Kof(case, dtype):
    return _K(case["nx"], case["ny"], case["nz"], dtype, case.get("Lz"))


def _forcing(K, gen, dtype):
    return [x[0] for x in _solenoidal(K, gen, dtype, lo=1.5, hi=3.5, slope=0.0)]


def _flow_inputs(case, seed):
    dt = _rdtype(case["prec"])
    K = _Kof(case, dt)
    gen = _gen(seed)
    v = [x[0] for x in _solenoidal(K, gen, dt)]
    f = _forcing(K, gen, dt) if case["forced"] else None
    a = th = None
    if case["kind"] == "mhd":
        a = [x[0] for x in _solenoidal(K, gen, dt, slope=-17.0 / 6.0, power=0.1)]
    if case["kind"] == "bouss":
        th = _spectrum(K, gen, dt, 1, 0.5, 1e9, -11.0 / 6.0)[0]
        e = (K.w * (th.real ** 2 + th.imag ** 2)).sum(dtype=torch.float64) / K.N ** 2
        th = (th * (0.01 / e).sqrt().to(dt)).contiguous()
    return v, f, a, th


def _ens_classes(case):
    return [(case["n%d" % q], case["r%d" % q]) for q in range(3)]


def _ens_inputs(case, seed):
    dt = _rdtype(case["prec"])
    gen = _gen(seed)
    rng = np.random.default_rng(seed)
    out = []
    for n, r in _ens_classes(case):
        v = _solenoidal(_K(n, n, n, dt), gen, dt, runs=r)
        out.append((v, np.exp(rng.uniform(math.log(5e-4), math.log(5e-3), r))))
    return out


def _mlp_params(seed):
    rng = np.random.default_rng(int(seed) + 17)
    glorot = lambda o, i: rng.uniform(-1, 1, (o, i)) * math.sqrt(6.0 / (o + i))  # noqa: E731
    small = lambda o: 0.1 * rng.standard_normal(o)  # noqa: E731
    p = [glorot(NHID, NIN), small(NHID), glorot(NHID, NHID), small(NHID), glorot(NOUT, NHID), small(NOUT)]
    return np.concatenate([q.ravel() for q in p]).astype(np.float32)


def _rows(case, seed, steps):
    """Minibatches of closure inputs (nine gradients of unit size and the
    filter width) and stress-like targets (quadratic in them)."""
    gen = _gen(seed, 5)
    B = case["batch"]
    x = torch.randn((steps, B, NIN), dtype=torch.float32, device=DEV, generator=gen)
    x[..., NIN - 1] = 1.0
    mix = torch.randn((9, NOUT), dtype=torch.float32, device=DEV, generator=gen) / 3.0
    t = (x[..., :9] @ mix) * x[..., :NOUT] * 0.6 + 0.3 * torch.randn((steps, B, NOUT), dtype=torch.float32, device=DEV,
                                                                     generator=gen)
    return x.contiguous(), t.contiguous()


# the closure's scales in an LES run
GRAD_SCALE, TAU_SCALE = 0.1, 0.02


def _les_inputs(case, seed):
    dt = _rdtype(case["prec"])
    K = _K(case["n"], case["n"], case["n"], dt)
    K.mask = (K.kk2 <= float(case["kc"] ** 2)) & (K.kk2 > 0)
    gen = _gen(seed)
    v = [x[0] for x in _solenoidal(K, gen, dt)]
    return v, _forcing(K, gen, dt)


# the physical parameters of the runs
HD_PAR = dict(dt=5e-4, nu=1e-3)
MHD_PAR = dict(dt=5e-4, nu=1e-3, mu=1e-3)
BOUSS_PAR = dict(dt=2.5e-4, nu=5e-4, kappa=5e-4, omegaz=0.5, xmom=8.0, xtemp=8.0)
ENS_DT = 1e-3
LES_PAR = dict(dt=2e-3, nu=1e-3)


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case = case
    kind = case["kind"]
    if kind in ("hd", "bouss", "mhd"):
        box = (1.0, 1.0, case["Lz"], True) if kind == "bouss" else ()
        s.g = Ghost(case["nx"], case["ny"], case["nz"], *box, precision=case["prec"])
        s.v, s.f, s.a, s.th = _flow_inputs(case, seed)
    elif kind == "ens":
        cls = _ens_classes(case)
        s.ens = Ensemble([n for n, _ in cls], [r for _, r in cls], precision=case["prec"])
        s.fields = [s.ens.fields(q) for q in range(3)]
        for q, (v, nu) in enumerate(_ens_inputs(case, seed)):
            n, r = cls[q]
            for dst, src in zip(s.fields[q], v):
                dst.copy_(src.view(r * (n // 2 + 1), n, n))
                dst.owner = s.ens  # the tensors view memory of the ensemble: it lives as long as they do
            s.ens.class_ctx(q).batch_set_nu(nu)
        torch.cuda.synchronize()  # the ensemble runs on streams of its own
    elif kind == "fft":
        s.g = Ghost(case["nx"], case["ny"], case["nz"], precision=case["prec"])
        n = (case["nx"], case["ny"], case["nz"])
        s.fwd = s.g.fftp3d_create_plan(n, GHOST_REAL_TO_COMPLEX)
        s.inv = s.g.fftp3d_create_plan(n, GHOST_COMPLEX_TO_REAL)
        s.r = torch.randn(s.g.rshape, dtype=s.g.rtorch, device=DEV, generator=_gen(seed))
        K = _Kof(case, s.g.rtorch)
        s.c = _spectrum(K, _gen(seed, 1), s.g.rtorch, 1, 0.5, 1e9, 0.0)[0]
        s.rc, s.cr = s.g.czeros(), s.g.rzeros()
    elif kind == "diag":
        s.g = Ghost(case["nx"], case["ny"], case["nz"], precision=case["prec"])
        K, gen = _Kof(case, s.g.rtorch), _gen(seed)
        s.v = [x[0] for x in _solenoidal(K, gen, s.g.rtorch)]
        s.f = _forcing(K, gen, s.g.rtorch)
        s.p = [s.g.czeros() for _ in range(3)]
        s.nl = [s.g.czeros() for _ in range(3)]
    elif kind in ("train", "infer"):
        s.mlp = MLP(0)
        s.mlp.params = _mlp_params(seed)
        s.x, s.t = _rows(case, seed, case.get("steps", 1))
    else:
        s.g = Ghost(case["n"], precision=case["prec"])
        s.les = LES(s.g, case["kc"])
        s.v, s.f = _les_inputs(case, seed)
        s.mlp = None
        if case["closure"].startswith("mlp"):
            s.mlp = MLP(0)
            s.mlp.params = _mlp_params(seed)
        s.les.set_model(case["closure"], s.mlp, grad_scale=GRAD_SCALE, tau_scale=TAU_SCALE, delta=1.0)
        s.les.set_time(1.0)
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "hd":
        s.g.hd_run(case["steps"], case["ord"], HD_PAR["dt"], HD_PAR["nu"], *s.v, *(s.f or ()))
        return s.v
    if kind == "bouss":
        p = BOUSS_PAR
        s.g.bouss_run(case["steps"], case["ord"], p["dt"], p["nu"], p["kappa"], p["omegaz"], p["xmom"], p["xtemp"],
                      *s.v, s.th, *(s.f or ()))
        return [*s.v, s.th]
    if kind == "mhd":
        p = MHD_PAR
        s.g.mhd_run(case["steps"], case["ord"], p["dt"], p["nu"], p["mu"], *s.v, *s.a, f=s.f or (None, None, None))
        return [*s.v, *s.a]
    if kind == "ens":
        s.ens.run(case["steps"], case["ord"], ENS_DT)
        return s.fields
    if kind == "fft":
        s.g.fftp3d_real_to_complex(s.fwd, s.r, s.rc)
        s.g.fftp3d_complex_to_real(s.inv, s.c, s.cr)
        return [s.rc, s.cr]
    if kind == "diag":
        g, v = s.g, s.v
        glob = g.hdcheck(*v, *s.f, 1, 0)
        vmax, wmax = g.maxabs(*v, 2), g.maxabs(*v, 0)
        Ek, Hk = g.spectrumc(*v, 1, 1)
        g.prodre3(*v, *s.p)
        for d in range(3):
            g.nonlhd3(*s.p, s.nl[d], d + 1)
        Tk = g.entrans(*v, *s.nl, 1)
        return {"eng": glob["eng"], "ens": glob["ens"], "khe": glob["khe"], "pot": glob["pot"], "vmax": vmax,
                "wmax": wmax, "Ek": Ek, "Hk": Hk, "Tk": Tk, "nl": s.nl}
    if kind == "train":
        for q in range(case["steps"]):
            s.mlp.train_step(s.x[q], s.t[q], 2e-3, want_loss=False)
        return s.mlp.params
    if kind == "infer":
        return s.mlp.forward(s.x[0])
    s.les.run(case["steps"], case["ord"], LES_PAR["dt"], LES_PAR["nu"], *s.v, *s.f)
    return s.v


# ---------------------------------------------------------------- what it takes
def _sizes(case):
    """(bytes of a spectral field, bytes of a real field, flops of one 3D transform)."""
    nx, ny, nz = (case["n"],) * 3 if "n" in case else (case["nx"], case["ny"], case["nz"])
    es = 4 if case["prec"] == "fp32" else 8
    N = nx * ny * nz
    return (nx // 2 + 1) * ny * nz * 2 * es, N * es, 2.5 * N * math.log2(N)


MLP_FLOP = 2 * (NIN * NHID + NHID * NHID + NHID * NOUT)


def work(case):
    kind = case["kind"]
    if kind == "ens":
        b = fl = 0.0
        for n, r in _ens_classes(case):
            C, _, T = _sizes(dict(n=n, prec=case["prec"]))
            b += 6 * C * r
            fl += 9 * T * r * case["ord"] * case["steps"]
        return {"bytes": b, "flops": fl}
    if kind == "train":
        rows = case["batch"] * case["steps"]
        return {"bytes": rows * 4 * (NIN + NOUT), "flops": rows * 3 * MLP_FLOP}
    if kind == "infer":
        return {"bytes": case["batch"] * 4 * (NIN + NOUT), "flops": case["batch"] * MLP_FLOP}
    C, R, T = _sizes(case)
    sub = case.get("ord", 1) * case.get("steps", 1)
    if kind == "hd":  # v in and out, the forcing in; nine transforms a substep
        return {"bytes": (9 if case["forced"] else 6) * C, "flops": 9 * T * sub}
    if kind == "bouss":
        return {"bytes": (11 if case["forced"] else 8) * C, "flops": 13 * T * sub}
    if kind == "mhd":
        return {"bytes": (15 if case["forced"] else 12) * C, "flops": 21 * T * sub}
    if kind == "fft":
        return {"bytes": 2 * (C + R), "flops": 2 * T}
    if kind == "diag":  # v and f in, the nonlinear term out; maxabs 2 x 3 and prodre3 9 transforms
        return {"bytes": 9 * C, "flops": 15 * T}
    mlp = case["n"] ** 3 * MLP_FLOP + 15 * T if case["closure"] == "mlp" else 0
    return {"bytes": 9 * C, "flops": (9 * T + mlp) * sub}


def tolerance(case):
    """About four times the error against 64 bits that was measured: what
    another order of rounding at the same precision can show.  `max` is a
    pointwise bound, over the field's root mean square."""
    kind, single = case["kind"], case.get("prec") == "fp32"
    if kind == "train":  # BF16 operands, and an Adam step turns a small gradient's sign into a step: 9e-4 seen
        return {"rel": 4e-3, "max": 0.3}
    if kind == "infer":  # BF16 operands
        return {"rel": 1e-2, "max": 0.2}
    if kind == "les" and case["closure"].startswith("mlp"):  # the BF16 network's force, times dt: 2.6e-7 seen
        return {"rel": 2e-6, "max": 1e-3}
    if kind == "les" and case["closure"] == "edqnm":  # the energy correction divides small differences
        return {"rel": 1e-5 if single else 1e-10, "max": 1e-2}
    if kind == "fft":  # 2.9e-7, 4.2e-16 seen
        return {"rel": 1.2e-6 if single else 2e-15, "max": 2e-5 if single else 3e-14}
    if kind == "diag":  # 6.2e-7 seen; sums of signed terms are conditioned worse
        return {"rel": 1e-5 if single else 1e-13, "max": 1e-3 if single else 1e-11}
    # steps: 5e-8, 8e-18 seen after one (an update is small beside the field), up to three are compared
    return {"rel": 5e-7 if single else 1e-15, "max": 1e-4 if single else 1e-12}


# ------------------------------------------------------------- 64-bit reference
def _real(K, a):
    nx, ny, nz = K.n
    return torch.fft.irfftn(a.permute(0, 3, 2, 1), s=(nz, ny, nx), dim=(1, 2, 3), norm="forward")


def _spec(r):
    return torch.fft.rfftn(r, dim=(1, 2, 3)).permute(0, 3, 2, 1)


def _curl(K, v):
    return [1j * (K.k[(q + 1) % 3] * v[(q + 2) % 3] - K.k[(q + 2) % 3] * v[(q + 1) % 3]) for q in range(3)]


def _cross(K, a, b):
    """Spectra of (a x b)/N^2 for the unnormalised real fields of two spectral triplets."""
    ra, rb = [_real(K, x) for x in a], [_real(K, x) for x in b]
    out = []
    for q in range(3):
        i, j = (q + 1) % 3, (q + 2) % 3
        out.append(_spec((ra[i] * rb[j] - ra[j] * rb[i]) / K.N ** 2))
    return out


def _minus_project(K, x):
    k2 = torch.where(K.kk2 > 0, K.kk2, torch.ones_like(K.kk2))
    s = (K.k[0] * x[0] + K.k[1] * x[1] + K.k[2] * x[2]) / k2
    return [K.k[q] * s - x[q] for q in range(3)]


def _hd_steps(K, v, f, steps, ord, dt, nu, force=None):
    """hd_run on (runs, nx/2+1, ny, nz) fields; nu a number or per run."""
    for _ in range(steps):
        C = [x.clone() for x in v]
        for o in range(ord, 0, -1):
            g = _minus_project(K, _cross(K, _curl(K, v), v))
            extra = force(v) if force else None
            for q in range(3):
                rhs = g[q] - nu * K.kk2 * v[q]
                if f is not None:
                    rhs = rhs + f[q]
                if extra is not None:
                    rhs = rhs + extra[q]
                v[q] = torch.where(K.mask, C[q] + dt / o * rhs, torch.zeros_like(rhs))
    return v


def _up(xs):
    return [x.to(torch.complex128)[None] for x in xs] if xs is not None else None


def _exact_bouss(case, K, v, th, f):
    p = BOUSS_PAR
    for _ in range(case["steps"]):
        C, C20 = [x.clone() for x in v], th.clone()
        for o in range(case["ord"], 0, -1):
            rv = [_real(K, x) for x in v]
            adv = sum(rv[q] * _real(K, 1j * K.k[q] * th) for q in range(3))
            del rv
            adv = _spec(-adv / K.N ** 2)
            g = _cross(K, _curl(K, v), v)
            g = [g[0] - 2 * p["omegaz"] * v[1], g[1] + 2 * p["omegaz"] * v[0], g[2] + p["xmom"] * th]
            g = _minus_project(K, g)
            r = p["dt"] / o
            nth = C20 + r * (adv + p["xtemp"] * v[2] - p["kappa"] * K.kk2 * th)
            # theta keeps its mean; the truncation zeroes the rest
            keep = K.mask | (K.kk2 == 0)
            th_old0 = C20[..., 0, 0, 0].clone()
            nth = torch.where(keep, nth, torch.zeros_like(nth))
            nth[..., 0, 0, 0] = th_old0
            for q in range(3):
                rhs = g[q] - p["nu"] * K.kk2 * v[q] + (f[q] if f is not None else 0)
                v[q] = torch.where(K.mask, C[q] + r * rhs, torch.zeros_like(rhs))
            th = nth
            del g, adv
    return [x[0] for x in v] + [th[0]]


def _exact_mhd(case, K, v, a, f):
    p = MHD_PAR
    for _ in range(case["steps"]):
        Cv, Ca = [x.clone() for x in v], [x.clone() for x in a]
        for o in range(case["ord"], 0, -1):
            b = _curl(K, a)
            wv, jb = _cross(K, _curl(K, v), v), _cross(K, _curl(K, b), b)
            g = _minus_project(K, [x - y for x, y in zip(wv, jb)])
            del wv, jb
            h = [-x for x in _minus_project(K, _cross(K, v, b))]
            for q in range(3):
                rv = g[q] - p["nu"] * K.kk2 * v[q] + (f[q] if f is not None else 0)
                ra = h[q] - p["mu"] * K.kk2 * a[q]
                v[q] = torch.where(K.mask, Cv[q] + p["dt"] / o * rv, torch.zeros_like(rv))
                a[q] = torch.where(K.mask, Ca[q] + p["dt"] / o * ra, torch.zeros_like(ra))
    return [x[0] for x in v + a]


def _shells(case, K, terms):
    """Shell sums, binned as the working precision bins (int(k/Dk + .501))."""
    kk = K.kk2.to(_rdtype(case["prec"])).sqrt()
    kmn = (kk / K.Dkk + kk.new_tensor(0.501, dtype=torch.float32).to(kk.dtype)).to(torch.int64)
    ok = (kmn > 0) & (kmn <= K.nbins)
    idx = torch.where(ok, kmn - 1, torch.full_like(kmn, K.nbins)).reshape(-1)
    out = torch.zeros(K.nbins + 1, dtype=torch.float64, device=DEV)
    out.index_add_(0, idx, (K.w * terms).reshape(-1))
    return out[:K.nbins].cpu().numpy()


def _exact_diag(case, K, v, f):
    dot = lambda a, b: sum((x.conj() * y).real for x, y in zip(a, b))[0] / K.N ** 2  # noqa: E731
    w = _curl(K, v)
    tot = lambda t: float((K.w * t).sum())  # noqa: E731
    vmax = float(sum(_real(K, x) ** 2 for x in v).sqrt().max()) / K.N
    wmax = float(sum(_real(K, x) ** 2 for x in w).sqrt().max()) / K.N
    nl = _minus_project(K, _cross(K, w, v))
    return {"eng": tot(dot(v, v)), "ens": tot(dot(w, w)), "khe": tot(dot(v, w)), "pot": tot(dot(v, f)), "vmax": vmax,
            "wmax": wmax, "Ek": _shells(case, K, dot(v, v)), "Hk": _shells(case, K, dot(v, w)),
            "Tk": _shells(case, K, dot(v, nl)), "nl": [x[0] for x in nl]}


def _unpack(p):
    out, o = [], 0
    for sh in ((NHID, NIN), (NHID,), (NHID, NHID), (NHID,), (NOUT, NHID), (NOUT,)):
        n = int(np.prod(sh))
        out.append(p[o:o + n].view(sh))
        o += n
    return out


C_GELU, A_GELU = math.sqrt(2.0 / math.pi), 0.044715


def _gelu(z):
    return 0.5 * z * (1 + torch.tanh(C_GELU * (z + A_GELU * z ** 3)))


def _gelu_d(z):
    t = torch.tanh(C_GELU * (z + A_GELU * z ** 3))
    return 0.5 * (1 + t) + 0.5 * z * (1 - t * t) * C_GELU * (1 + 3 * A_GELU * z * z)


def _mlp64(p, x):
    W1, b1, W2, b2, W3, b3 = _unpack(p)
    z1 = x @ W1.T + b1
    h1 = _gelu(z1)
    z2 = h1 @ W2.T + b2
    h2 = _gelu(z2)
    return h2 @ W3.T + b3, (z1, h1, z2, h2, W2, W3)


def _exact_train(case, seed):
    p = torch.tensor(_mlp_params(seed), device=DEV).double()
    X, T = _rows(case, seed, case["steps"])
    m, s = torch.zeros_like(p), torch.zeros_like(p)
    for q in range(case["steps"]):
        x, t = X[q].double(), T[q].double()
        y, (z1, h1, z2, h2, W2, W3) = _mlp64(p, x)
        dy = (y - t) * (2.0 / (x.shape[0] * NOUT))
        d2 = (dy @ W3) * _gelu_d(z2)
        d1 = (d2 @ W2) * _gelu_d(z1)
        g = torch.cat([(d1.T @ x).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1), d2.sum(0), (dy.T @ h2).reshape(-1),
                       dy.sum(0)])
        m = 0.9 * m + 0.1 * g
        s = 0.999 * s + 0.001 * g * g
        p = p - 2e-3 * (m / (1 - 0.9 ** (q + 1))) / ((s / (1 - 0.999 ** (q + 1))).sqrt() + 1e-8)
    return p.cpu().numpy()


def _exact_les(case, seed):
    v, f = _les_inputs(case, seed)
    K = _K(case["n"], case["n"], case["n"], torch.float64)
    K.mask = (K.kk2 <= float(case["kc"] ** 2)) & (K.kk2 > 0)
    v, f = _up(v), _up(f)
    force = None
    if case["closure"] == "mlp":
        p = torch.tensor(_mlp_params(seed), device=DEV).double()
        slot = ((0, 3, 4), (3, 1, 5), (4, 5, 2))

        def force(v):
            gr = [_real(K, 1j * K.k[b] * v[a]) / K.N * GRAD_SCALE for a in range(3) for b in range(3)]
            x = torch.stack(gr + [torch.ones_like(gr[0])], dim=-1).reshape(-1, NIN)
            del gr
            y = torch.cat([_mlp64(p, q)[0] for q in x.split(1 << 18)]) * TAU_SCALE
            n = case["n"]
            T = [_spec(y[:, m].reshape(1, n, n, n)) for m in range(NOUT)]
            F = [sum(-1j * K.k[b] * T[slot[a][b]] for b in range(3)) for a in range(3)]
            return [torch.where(K.mask, -q, torch.zeros_like(q)) for q in _minus_project(K, F)]

    v = _hd_steps(K, v, f, case["steps"], case["ord"], LES_PAR["dt"], LES_PAR["nu"], force)
    return [x[0] for x in v]


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "infer":
        p = torch.tensor(_mlp_params(seed), device=DEV).double()
        x, _ = _rows(case, seed, 1)
        return torch.cat([_mlp64(p, q.double())[0] for q in x[0].split(1 << 18)])
    if kind == "les":
        # the eddy-viscosity closures fit and integrate spectra: no short statement of them here
        return _exact_les(case, seed) if case["closure"] in ("none", "mlp") else None
    if kind == "ens":
        out = []
        for (n, r), (v, nu) in zip(_ens_classes(case), _ens_inputs(case, seed)):
            K = _K(n, n, n, torch.float64)
            v = [x.to(torch.complex128) for x in v]
            nu = torch.tensor(nu, device=DEV).view(-1, 1, 1, 1)
            v = _hd_steps(K, v, None, case["steps"], case["ord"], ENS_DT, nu)
            out.append([x.reshape(r * (n // 2 + 1), n, n) for x in v])
        return out
    K = _Kof(case, torch.float64)
    if kind == "fft":
        dt = _rdtype(case["prec"])
        r = torch.randn((case["nz"], case["ny"], case["nx"]), dtype=dt, device=DEV, generator=_gen(seed))
        c = _spectrum(_Kof(case, dt), _gen(seed, 1), dt, 1, 0.5, 1e9, 0.0)
        return [_spec(r.double()[None])[0], _real(K, c.to(torch.complex128))[0]]
    if kind == "diag":
        dt = _rdtype(case["prec"])
        Kp, gen = _Kof(case, dt), _gen(seed)
        v = [x[0] for x in _solenoidal(Kp, gen, dt)]
        f = _forcing(Kp, gen, dt)
        return _exact_diag(case, K, _up(v), _up(f))
    v, f, a, th = _flow_inputs(case, seed)
    v, f = _up(v), _up(f)
    if kind == "bouss":
        return _exact_bouss(case, K, v, th.to(torch.complex128)[None], f)
    if kind == "mhd":
        return _exact_mhd(case, K, v, _up(a), f)
    return [x[0] for x in _hd_steps(K, v, f, case["steps"], case["ord"], HD_PAR["dt"], HD_PAR["nu"])]
