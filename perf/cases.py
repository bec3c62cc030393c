"""Timed cases of the framework: what its users have it do, through its public
entry points, over the range of sizes, precisions and options in use.

Kinds of pass:

``step``       ``k`` time steps of a resident model (``SHTnsKitConfig.step``), then its
               fields copied to the caller's device buffers, as a run does between
               two outputs.  All precision settings; CNAB2 and EAB2; with and
               without composition.
``synth``      scalar synthesis of fields that live on the device in a solver loop
               that allocates nothing (``gd_spectral_to_physical_noalloc``).
``roundtrip``  vector synthesis and analysis on host arrays, the drop-in use by a
               program that keeps its fields itself (``shtnskit_vector_synthesis``,
               ``shtnskit_vector_analysis``).
``ensemble``   ``k`` steps of a batch of uneven shells (``Ensemble``), then all fields.
``gradient``   ``k`` checkpointed steps and the gradient of a functional of the final
               temperature with respect to the initial temperature and velocity
               (``temperature_forward``, ``temperature_pullback_full``).

A mixed-precision model computes its nonlinear terms in FP32, so its caller
keeps FP32 copies of those fields; the velocity of the ``mixed_vel64*`` settings
and every field of an FP64 model are FP64.
"""
import functools
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FIELDS = ("u_tor", "u_pol", "b_tor", "b_pol", "temp", "comp")
PHYSICS = dict(rratio=0.35, ekman=3e-4, prandtl=1.0, magnetic_prandtl=4.0, implicit_theta=0.5)
KL = 4


def _package():
    """The framework's package (its directory's name is not a Python identifier)."""
    if "gdb200" not in sys.modules:
        pkg = os.path.join(ROOT, "geodynamo.jl_b200")
        spec = importlib.util.spec_from_file_location("gdb200", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["gdb200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["gdb200"]


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _step(lmax, nlat, nlon, nr, precision, k, dt, composition=0, scheme="cnab2"):
    return dict(kind="step", lmax=lmax, nlat=nlat, nlon=nlon, nr=nr, precision=precision, k=k, dt=dt,
                composition=composition, scheme=scheme)


def listed():
    return [
        # one field on 32 shells: the smallest call, a few microseconds of kernels behind a launch
        dict(name="synth_l31_nr32", kind="synth", lmax=31, nlat=48, nlon=96, nr=32, nfield=1),
        # a batch of nine fields at the transform benchmark's angular grid (lmax 127), a third of its shells
        dict(name="synth_l127_nr33x9", kind="synth", lmax=127, nlat=192, nlon=384, nr=33, nfield=9),
        # drop-in vector transforms on host arrays, default grid of create_shtnskit_config (nlat = lmax + 3)
        dict(name="roundtrip_l85_nr33", kind="roundtrip", lmax=85, nlat=88, nlon=180, nr=33),
        # the oracle configuration in FP64: small, bound by launches and latency
        dict(_step(31, 48, 96, 32, "fp64", 10, 1e-5), name="step_fp64_l31_nr32"),
        # fast mixed step on the default grid (no 3/2 dealiasing): nlat = lmax + 3, nlon = 256
        dict(_step(127, 130, 256, 65, "mixed", 4, 5e-6), name="step_mixed_l127_nr65"),
        # ragged sizes with composition, velocity chain in FP64
        dict(_step(140, 212, 288, 97, "mixed_vel64", 4, 4e-6, composition=1), name="step_vel64_l140_nr97"),
        # exponential scheme at the adjoint configuration's grid
        dict(_step(63, 96, 192, 65, "fp64", 4, 1e-6, scheme="eab2"), name="step_eab2_l63_nr65"),
        # all-FP64 step at the headline's angular grid
        dict(_step(255, 384, 768, 33, "fp64", 2, 2e-6), name="step_fp64_l255_nr33"),
        # the headline: velocity chain at FP64 accuracy by int8 slices
        dict(_step(255, 384, 768, 129, "mixed_vel64i8", 2, 2e-6), name="step_vel64i8_l255_nr129"),
        # a higher resolution with few shells per GPU, fast mixed
        dict(_step(341, 512, 1024, 33, "mixed", 2, 1e-6), name="step_mixed_l341_nr33"),
        # a batch of uneven shells, grouped by angular grid
        dict(name="ensemble_mixed_x12", kind="ensemble", members=12, precision="mixed", k=4, dt=2e-6),
        # gradient by checkpoint and recompute at the adjoint configuration's grid
        dict(name="gradient_l63_nr65", kind="gradient", lmax=63, nlat=96, nlon=192, nr=65, k=8, every=4, dt=5e-6),
    ]


def _smooth(n):
    while True:
        m = n
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _angular(rng, lmax):
    """The 3/2-rule grid or create_shtnskit_config's default grid."""
    if rng.random() < 0.5:
        nlat = 3 * (lmax + 1) // 2
        nlat += nlat & 1
        return nlat, _smooth(2 * nlat)
    nlat = lmax + 2
    nlat += nlat & 1
    return nlat, _smooth(2 * lmax + 1)


def draw(rng):
    kind = rng.choice(("step", "step", "step", "step", "synth", "roundtrip", "ensemble", "gradient"))
    if kind == "step":
        lmax = _log_int(rng, 21, 300)
        nr = _log_int(rng, 15, 129)
        # no more grid points than the headline (lmax 255, nr 129), fewer in FP64
        precision = rng.choice(("fp64", "mixed", "mixed_vel64", "mixed_vel64i8"))
        cap = (1.0 if precision != "fp64" else 0.4) * 0.8 * 255.0 ** 3 * 129 / lmax ** 3
        nr = max(9, min(nr, int(cap)))
        nlat, nlon = _angular(rng, lmax)
        return _step(lmax, nlat, nlon, nr, precision, 2 if lmax > 128 else 4, 2e-6,
                     composition=int(rng.random() < 0.25))
    if kind == "synth":
        lmax = _log_int(rng, 15, 150)
        nlat, nlon = _angular(rng, lmax)
        # four fields' Fourier coefficients fit the call's fixed 64 MiB
        most = (64 << 20) // (4 * (lmax + 1) * nlat * 16)
        return dict(kind="synth", lmax=lmax, nlat=nlat, nlon=nlon, nr=max(3, min(_log_int(rng, 5, 97), most)),
                    nfield=rng.randint(1, 9))
    if kind == "roundtrip":
        lmax = _log_int(rng, 21, 120)
        nlat, nlon = _angular(rng, lmax)
        return dict(kind="roundtrip", lmax=lmax, nlat=nlat, nlon=nlon, nr=_log_int(rng, 9, 49))
    if kind == "ensemble":
        return dict(kind="ensemble", members=rng.randint(3, 12), precision=rng.choice(("mixed", "fp64")), k=4,
                    dt=rng.choice((1e-6, 2e-6)))
    lmax = _log_int(rng, 21, 80)
    nlat, nlon = _angular(rng, lmax)
    k = rng.randint(2, 8)
    return dict(kind="gradient", lmax=lmax, nlat=nlat, nlon=nlon, nr=_log_int(rng, 12, 65), k=k,
                every=rng.randint(1, k), dt=2e-6)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _modes(lmax):
    """l and m of the native (m-major) mode order, the native index of each l-major mode."""
    l = np.concatenate([np.arange(m, lmax + 1) for m in range(lmax + 1)])
    m = np.concatenate([np.full(lmax + 1 - m, m) for m in range(lmax + 1)])
    return l, m, np.lexsort((m, l))


def _radial_nodes(nr):
    ri = PHYSICS["rratio"] / (1.0 - PHYSICS["rratio"])
    return ri + 0.5 * (1.0 + np.cos(np.pi * np.arange(nr - 1, -1, -1) / (nr - 1)))


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _random_field(gen, lmax, nr, amp, power, potential):
    """(2, nr, nlm) native planes: normal coefficients under a power-law spectrum and a
    radial profile that vanishes at the boundaries."""
    l, m, _ = _modes(lmax)
    r = _radial_nodes(nr)
    prof = torch.as_tensor(amp * np.sin(np.pi * (r - r[0]) / (r[-1] - r[0])), device="cuda")
    spec = torch.as_tensor((l + 1.0) ** -power, device="cuda")
    a = torch.randn(2, nr, l.size, generator=gen, device="cuda", dtype=torch.float64)
    a *= prof[:, None] * spec
    a[1][:, torch.as_tensor(m == 0, device="cuda")] = 0.0
    if potential:
        a[:, :, 0] = 0.0  # l = 0 carries no field
    return a


def _state(seed, lmax, nr, names):
    """A developed convective state: velocity of tens of diffusion units, temperature and
    composition perturbations of order one, a magnetic field of order one."""
    gen = _generator(seed)
    amp = dict(u_tor=10.0, u_pol=5.0, b_tor=1.0, b_pol=1.0, temp=0.5, comp=0.5)
    return {k: _random_field(gen, lmax, nr, amp[k], 2.0, k not in ("temp", "comp")) for k in names}


def _members(case):
    """Member configurations of an ensemble case, from the sizes of the batched uneven ensemble."""
    rng = np.random.default_rng(3)
    out = []
    for _ in range(case["members"]):
        lmax = int((31, 47, 63, 95)[rng.integers(4)])
        nr = int((33, 49, 65)[rng.integers(3)])
        nlat = 3 * (lmax + 1) // 2
        out.append(dict(lmax=lmax, nlat=nlat, nlon=2 * nlat, nr=nr, dt=case["dt"], bc_mode=2, kl=KL,
                        **dict(PHYSICS, ekman=float(10.0 ** rng.uniform(-4.0, -3.0)))))
    return out


def _names(case):
    return FIELDS if case.get("composition") else FIELDS[:5]


def _boundary_temperature(lmax):
    """Boundary values [2][nlm] (l-major): the inner sphere one unit warmer."""
    b = np.zeros((2, (lmax + 1) * (lmax + 2) // 2))
    b[0, 0] = math.sqrt(4.0 * math.pi)
    return b


class _Readout:
    """The caller's device buffers of a model's fields, and how they are filled."""

    def __init__(self, model, names, precision):
        self.model = model
        self.names = names
        self.buf = [torch.empty(2, model.nr, model.nlm, device="cuda", dtype=torch.float64) for _ in names]
        single = {"fp64": (), "mixed": names}.get(precision, names[2:])
        self.single = [n in single for n in names]

    def load(self, fields):
        for i, n in enumerate(self.names):
            self.model.copy_block(0, FIELDS.index(n), 0, self.model.nr, 0, self.model.nlm, fields[n].data_ptr(), False)

    def read(self):
        # copy_block fills the buffers on the model's stream and waits; the FP32 copies of
        # the read before, on torch's stream, must have left them
        if any(self.single):
            torch.cuda.current_stream().synchronize()
        for n, b in zip(self.names, self.buf):
            self.model.copy_block(0, FIELDS.index(n), 0, self.model.nr, 0, self.model.nlm, b.data_ptr(), True)
        return [b.float() if s else b for b, s in zip(self.buf, self.single)]


def prepare(case, seed):
    gdb = _package()
    kind = case["kind"]
    if kind == "ensemble":
        cfgs = _members(case)
        ens = gdb.Ensemble(cfgs, precision=case["precision"], group=64)
        # state of the members, packed per handle along r as the handle stacks them
        parts = [[] for _ in ens.handles]
        for i, (c, m) in enumerate(zip(cfgs, ens.members)):
            h = getattr(m, "handle", m)
            base = m.rows.start if hasattr(m, "rows") else 0
            parts[next(k for k, x in enumerate(ens.handles) if x is h)].append(
                (base, _state(seed * 64 + i, c["lmax"], c["nr"], FIELDS[:5])))
        outs = []
        for h, p in zip(ens.handles, parts):
            p.sort(key=lambda q: q[0])
            ro = _Readout(h, FIELDS[:5], case["precision"])
            torch.cuda.current_stream().synchronize()
            ro.load({n: torch.cat([s[n] for _, s in p], 1).contiguous() for n in FIELDS[:5]})
            outs.append(ro)
        return dict(case=case, ens=ens, outs=outs)
    args = dict(lmax=case["lmax"], nlat=case["nlat"], nlon=case["nlon"], nr=case["nr"], kl=KL, **PHYSICS)
    if kind == "synth":
        model = gdb.SHTnsKitConfig(**args)
        gen = _generator(seed)
        coef = torch.stack([_random_field(gen, case["lmax"], case["nr"], 1.0, 1.5, False)
                            for _ in range(case["nfield"])])
        grid = torch.empty(case["nfield"], case["nr"], case["nlat"], case["nlon"], device="cuda", dtype=torch.float64)
        torch.cuda.current_stream().synchronize()
        return dict(case=case, model=model, coef=coef, grid=grid)
    if kind == "roundtrip":
        model = gdb.SHTnsKitConfig(**args)
        gen = _generator(seed)
        tor, pol = gdb.SHTnsSpectralField(model), gdb.SHTnsSpectralField(model)
        order = _modes(case["lmax"])[2]
        for f in (tor, pol):
            a = _random_field(gen, case["lmax"], case["nr"], 1.0, 1.5, True).cpu().numpy()
            f.data_real[...] = a[0][:, order]
            f.data_imag[...] = a[1][:, order]
        return dict(case=case, model=model, tor=tor, pol=pol, vec=gdb.SHTnsVectorField(model),
                    back=(gdb.SHTnsSpectralField(model), gdb.SHTnsSpectralField(model)))
    if kind == "gradient":
        model = gdb.SHTnsKitConfig(dt=case["dt"], bc_mode=2, **args)
        model.set_temperature_bc(_boundary_temperature(case["lmax"]))
        fields = _state(seed, case["lmax"], case["nr"], FIELDS[:5])
        gen = _generator(seed + (1 << 40))
        lam = _random_field(gen, case["lmax"], case["nr"], 1.0, 1.0, False).cpu().numpy()[:, :, _modes(case["lmax"])[2]]
        torch.cuda.current_stream().synchronize()
        out = _Readout(model, FIELDS[:5], "fp64")
        out.load(fields)
        return dict(case=case, model=model, out=out, lam=np.ascontiguousarray(lam))
    bc = 0 if case["scheme"] == "eab2" else 2
    model = gdb.SHTnsKitConfig(dt=case["dt"], bc_mode=bc, precision=case["precision"],
                               composition=case["composition"], **args)
    model.set_temperature_bc(_boundary_temperature(case["lmax"]))
    if case["scheme"] != "cnab2":
        model.set_scheme(case["scheme"])
    fields = _state(seed, case["lmax"], case["nr"], _names(case))
    out = _Readout(model, _names(case), case["precision"])
    torch.cuda.current_stream().synchronize()
    out.load(fields)
    # the exponential scheme's operators carry no boundary rows and grow without
    # bound, so its runs are short ones from a kept state
    return dict(case=case, model=model, out=out, start=fields if bc == 0 else None)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "step":
        if state["start"] is not None:
            state["out"].load(state["start"])
        state["model"].step(case["k"])
        return state["out"].read()
    if kind == "synth":
        model = state["model"]
        model._check(model.lib.gd_spectral_to_physical_noalloc(model.h, case["nfield"], state["coef"].data_ptr(),
                                                               state["grid"].data_ptr()))
        model.synchronize()  # the result is used on the caller's stream
        return state["grid"]
    if kind == "roundtrip":
        gdb = _package()
        vec, (tor, pol) = state["vec"], state["back"]
        gdb.shtnskit_vector_synthesis(state["tor"], state["pol"], vec)
        gdb.shtnskit_vector_analysis(vec, tor, pol)
        return [vec.theta_component.data, vec.phi_component.data, tor.data_real, tor.data_imag, pol.data_real,
                pol.data_imag]
    if kind == "ensemble":
        state["ens"].step(case["k"])
        return [o.read() for o in state["outs"]]
    model = state["model"]
    model.temperature_forward(case["k"], case["every"])
    gradient = model.temperature_pullback_full(state["lam"][0], state["lam"][1])
    return dict(gradient=gradient, fields=state["out"].read())


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _legendre_flops(lmax, nlat, vec):
    """One transform of one shell, north/south folding used: complex coefficients on half the latitudes."""
    nlm = (lmax + 1) * (lmax + 2) / 2
    return (4 if vec else 1) * 4 * nlm * (nlat / 2)


def _fft_flops(nlat, nlon):
    return nlat * 2.5 * nlon * math.log2(nlon)


def _step_work(lmax, nlat, nlon, nr, k, comp, scheme="cnab2"):
    nlm = (lmax + 1) * (lmax + 2) / 2
    nf = 6 if comp else 5
    scalar, vec = _legendre_flops(lmax, nlat, False), _legendre_flops(lmax, nlat, True)
    fft = _fft_flops(nlat, nlon)
    # per step: temperature (and composition) 4 syntheses and 1 analysis; u, curl u, B, curl B
    # syntheses and 2 vector analyses; the radial solves
    flops = (1 + comp) * (5 * (scalar + fft)) + 6 * (vec + 2 * fft) + nf * nlm * 2 * (2 * 9 + 2 * 9)
    if scheme != "cnab2":
        flops += nf * nlm * 2 * 2 * 2 * nr
    # fields in and out, the terms of two steps in and one out
    return dict(bytes=k * nf * 5 * 2 * nr * nlm * 8.0, flops=float(k * nr * flops))


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        parts = [_step_work(c["lmax"], c["nlat"], c["nlon"], c["nr"], case["k"], 0) for c in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    lmax, nlat, nlon, nr = case["lmax"], case["nlat"], case["nlon"], case["nr"]
    nlm = (lmax + 1) * (lmax + 2) / 2
    if kind == "synth":
        n = case["nfield"] * nr
        return dict(bytes=n * 8.0 * (2 * nlm + nlat * nlon) + nlm * nlat / 2 * 8.0,
                    flops=float(n * (_legendre_flops(lmax, nlat, False) + _fft_flops(nlat, nlon))))
    if kind == "roundtrip":
        # coefficients in, two grids out and in, coefficients out
        return dict(bytes=nr * 8.0 * (4 * nlm + 4 * nlat * nlon + 4 * nlm),
                    flops=float(nr * 2 * (_legendre_flops(lmax, nlat, True) + 2 * _fft_flops(nlat, nlon))))
    if kind == "gradient":
        w = _step_work(lmax, nlat, nlon, nr, case["k"], 0)
        # a forward run, its recomputation, and a transposed step for each
        return {k: 3 * v for k, v in w.items()}
    return _step_work(lmax, nlat, nlon, nr, case["k"], case["composition"], case["scheme"])


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
class _Exact:
    """Spherical-harmonic transforms on dense (m, l, theta) tables.  Coefficients are complex
    (nr, m, l), grids (nr, theta, phi)."""

    def __init__(self, lmax, nlat, nlon):
        self.lmax, self.nlat, self.nlon = lmax, nlat, nlon
        x, w = self._gauss(nlat)
        th = np.arccos(x)
        self.ct = torch.as_tensor(x, device="cuda")
        self.w = torch.as_tensor(w, device="cuda")
        sn = torch.as_tensor(np.sin(th), device="cuda")
        L = lmax
        m = torch.arange(L + 2, device="cuda", dtype=torch.float64)[:, None]
        P = torch.zeros(L + 2, L + 1, nlat, device="cuda", dtype=torch.float64)  # one order more, for dP at m = 0
        pmm = torch.full((nlat,), 1.0 / math.sqrt(4.0 * math.pi), device="cuda", dtype=torch.float64)
        for l in range(L + 1):
            if l:
                pmm = -math.sqrt((2.0 * l + 1.0) / (2.0 * l)) * sn * pmm
            P[l, l] = pmm
            if l:
                P[l - 1, l] = math.sqrt(2.0 * l + 1.0) * self.ct * P[l - 1, l - 1]
            if l > 1:
                mm = m[:l - 1]
                a = torch.sqrt((4.0 * l * l - 1.0) / (l * l - mm * mm))
                b = torch.sqrt(((l - 1.0) ** 2 - mm * mm) / (4.0 * (l - 1.0) ** 2 - 1.0))
                P[:l - 1, l] = a * (self.ct * P[:l - 1, l - 1] - b * P[:l - 1, l - 2])
        l = torch.arange(L + 1, device="cuda", dtype=torch.float64)[None, :]
        mm = m[:L + 1]
        cf = torch.sqrt(torch.clamp((2.0 * l + 1.0) * (l * l - mm * mm) / (2.0 * l - 1.0), min=0.0))
        prev = torch.zeros_like(P[:L + 1])
        prev[:, 1:] = P[:L + 1, :-1]
        dP = (l[..., None] * self.ct * P[:L + 1] - cf[..., None] * prev) / sn
        dP[0] = torch.sqrt(l[0] * (l[0] + 1.0))[:, None] * P[1]
        self.P = P[:L + 1].contiguous()
        self.dP = dP
        self.Q = mm[..., None] * self.P / sn
        self.l, self.m = l[0], mm[:, 0]

    @staticmethod
    def _gauss(n):
        """Gauss-Legendre nodes from north to south: Newton steps in theta."""
        t = np.pi * (np.arange(1, n + 1) - 0.25) / (n + 0.5)
        for _ in range(8):
            x, s = np.cos(t), np.sin(t)
            p0, p1 = np.ones_like(x), x.copy()
            for k in range(2, n + 1):
                p0, p1 = p1, ((2.0 * k - 1.0) * x * p1 - (k - 1.0) * p0) / k
            q = n * (p0 - x * p1)  # (1 - x^2) P_n'
            t = t + p1 * s / q
        return np.cos(t), 2.0 * np.sin(t) ** 2 / (q * q)

    def _leg(self, a, tab):  # (nr, m, l) -> (nr, theta, m)
        x = torch.view_as_real(a).permute(1, 0, 3, 2).reshape(self.lmax + 1, -1, self.lmax + 1)
        y = torch.bmm(x, tab).reshape(self.lmax + 1, a.shape[0], 2, self.nlat)
        return torch.complex(y[:, :, 0], y[:, :, 1]).permute(1, 2, 0)

    def _leg_t(self, g, tab):  # (nr, theta, m) -> (nr, m, l)
        x = torch.stack([g.real, g.imag], 0).permute(3, 1, 0, 2).reshape(self.lmax + 1, -1, self.nlat)
        y = torch.bmm(x, tab.transpose(1, 2)).reshape(self.lmax + 1, g.shape[0], 2, self.lmax + 1)
        return torch.complex(y[:, :, 0], y[:, :, 1]).permute(1, 0, 2)

    def _to_grid(self, F):
        return torch.fft.irfft(F, n=self.nlon, dim=2, norm="forward")

    def _from_grid(self, f):
        return torch.fft.rfft(f, dim=2)[..., :self.lmax + 1] * (2.0 * math.pi / self.nlon) * self.w[:, None]

    def _real_m0(self, a):
        keep = torch.ones(self.lmax + 1, 1, device="cuda", dtype=torch.float64)
        keep[0] = 0.0
        return torch.complex(a.real, a.imag * keep)

    def synth(self, a):
        return self._to_grid(self._leg(a, self.P))

    def analysis(self, f):
        return self._real_m0(self._leg_t(self._from_grid(f), self.P))

    def synth_vector(self, T, S):
        return (self._to_grid(self._leg(S, self.dP) + 1j * self._leg(T, self.Q)),
                self._to_grid(1j * self._leg(S, self.Q) - self._leg(T, self.dP)))

    def analysis_vector(self, vt, vp):
        gt, gp = self._from_grid(vt), self._from_grid(vp)
        f = 1.0 / torch.clamp(self.l * (self.l + 1.0), min=1.0)
        f = torch.where(self.l > 0, f, torch.zeros_like(f))
        S = self._leg_t(gt, self.dP) - 1j * self._leg_t(gp, self.Q)
        T = -1j * self._leg_t(gt, self.Q) - self._leg_t(gp, self.dP)
        return self._real_m0(T * f), self._real_m0(S * f)

    # packed native planes (2, nr, nlm) <-> dense
    def dense(self, planes):
        l, m, _ = _modes(self.lmax)
        z = torch.zeros(planes.shape[1], self.lmax + 1, self.lmax + 1, device="cuda", dtype=torch.complex128)
        r = torch.arange(planes.shape[1], device="cuda")[:, None]
        at = (r, torch.as_tensor(m, device="cuda")[None], torch.as_tensor(l, device="cuda")[None])
        return z.index_put(at, torch.complex(planes[0], planes[1]))

    def packed(self, a):
        l, m, _ = _modes(self.lmax)
        v = a[:, torch.as_tensor(m, device="cuda"), torch.as_tensor(l, device="cuda")]
        return torch.stack([v.real, v.imag])


@functools.lru_cache(maxsize=4)
def _exact_grid(lmax, nlat, nlon):
    return _Exact(lmax, nlat, nlon)


def _weights(r, order):
    """Dense difference matrix of stencils of up to 2 KL + 1 nodes (clipped at the ends)."""
    n = r.size
    D = np.zeros((n, n))
    for i in range(n):
        a, b = max(0, i - KL), min(n, i + KL + 1)
        V = np.vander(r[a:b] - r[i], increasing=True).T
        e = np.zeros(b - a)
        e[order] = 2.0 if order == 2 else 1.0
        D[i, a:b] = np.linalg.solve(V, e)
    return D


class _ExactModel:
    """The time step of a shell: advection of T (and C) by the velocity of the step before
    (this step's for C), the Coriolis term of u, no other nonlinear term in value (the
    synthesised vectors have no radial components), implicit diffusion."""

    def __init__(self, g, nr, dt, ekman, scheme="cnab2", bc_rows=True):
        self.g, self.dt, self.scheme, self.bc_rows = g, dt, scheme, bc_rows
        r = _radial_nodes(nr)
        self.r = torch.as_tensor(r, device="cuda")
        lap = torch.as_tensor(_weights(r, 2) + (2.0 / r)[:, None] * _weights(r, 1), device="cuda")
        ll = g.l * (g.l + 1.0)
        eye = torch.eye(nr, device="cuda", dtype=torch.float64)
        pm = PHYSICS["magnetic_prandtl"]
        nu = dict(u_tor=pm, u_pol=pm, b_tor=1.0, b_pol=1.0, temp=pm / PHYSICS["prandtl"], comp=pm)
        self.lin, self.imp, self.exp = {}, {}, {}
        for v in set(nu.values()):
            A = v * (lap[None] - ll[:, None, None] * torch.diag(1.0 / self.r ** 2)[None])
            self.lin[v] = A
            B = eye / dt - PHYSICS["implicit_theta"] * A
            if bc_rows:
                B[:, 0] = eye[0]
                B[:, -1] = eye[-1]
            self.imp[v] = torch.linalg.lu_factor(B)
            if scheme == "eab2":
                big = torch.zeros(A.shape[0], 2 * nr, 2 * nr, device="cuda", dtype=torch.float64)
                big[:, :nr, :nr] = dt * A
                big[:, :nr, nr:] = eye
                e = torch.linalg.matrix_exp(big)
                self.exp[v] = (e[:, :nr, :nr].contiguous(), e[:, :nr, nr:].contiguous())
        self.nu = nu
        self.rf = pm / ekman
        j = torch.clamp(torch.arange(g.nlon, device="cuda"), max=g.nlat - 1)
        self.cor = self.rf * g.ct[j]
        self.t0 = math.sqrt(4.0 * math.pi)
        self.grids = None
        self.prev = {}

    def _per_l(self, mats, a):  # (l, i, j) applied to (j, m, l)
        x = torch.view_as_real(a).permute(2, 0, 1, 3).reshape(a.shape[2], a.shape[0], -1)
        return self._back(torch.bmm(mats, x), a)

    @staticmethod
    def _back(y, a):
        y = y.reshape(a.shape[2], a.shape[0], a.shape[1], 2).permute(1, 2, 0, 3).contiguous()
        return torch.view_as_complex(y)

    def _solve(self, lu, a):
        x = torch.view_as_real(a).permute(2, 0, 1, 3).reshape(a.shape[2], a.shape[0], -1)
        return self._back(torch.linalg.lu_solve(*lu, x), a)

    def _rows(self, a, inner):
        """Fixed boundary values: `inner` at r_i for l = 0, zero elsewhere."""
        row = torch.zeros_like(a[0])
        first = row.clone()
        first[0, 0] = inner
        return torch.cat([first[None], a[1:-1], row[None]], 0)

    def _advect(self, a):
        g = self.g
        l, m = g.l[None, :], g.m[:, None]
        up = torch.cat([a[:, :, 1:], torch.zeros_like(a[:, :, :1])], 2)
        dn = torch.cat([torch.zeros_like(a[:, :, :1]), a[:, :, :-1]], 2)
        cp = torch.clamp((l + 1) ** 2 - m * m, min=0.0) / (2.0 * l + 1.0)
        cp = torch.where((l >= m) & (l + 1 <= g.lmax), cp, torch.zeros_like(cp))
        cm = torch.where(l - 1 >= m, -(l * l - m * m) / (2.0 * l - 1.0), torch.zeros_like(cp))
        ri = (1.0 / self.r)[:, None, None]
        gth = g.synth((cp * up + cm * dn) * ri)
        gph = g.synth(1j * m * a * ri)
        ut, up_ = self.grids
        return g.analysis(-(ut * gth + up_ * gph))

    def step(self, s):
        g = self.g
        n = {}
        if self.grids is None:
            z = torch.zeros(self.r.numel(), g.nlat, g.nlon, device="cuda", dtype=torch.float64)
            self.grids = (z, z)
        s = dict(s)
        n["temp"] = self._advect(s["temp"])
        s["temp"] = self._rows(s["temp"], self.t0)
        self.grids = g.synth_vector(s["u_tor"], s["u_pol"])
        n["u_tor"], n["u_pol"] = g.analysis_vector(self.cor * self.grids[1], -self.cor * self.grids[0])
        if "comp" in s:
            n["comp"] = self._advect(s["comp"])
            s["comp"] = self._rows(s["comp"], 0.0)
        out = {}
        for k, u in s.items():
            v = self.nu[k]
            nk = n.get(k)
            if self.scheme == "eab2":
                x = self._per_l(self.exp[v][0], u)
                if nk is not None:
                    x = x + self.dt * self._per_l(self.exp[v][1], 1.5 * nk - 0.5 * self.prev.get(k, torch.zeros_like(nk)))
            else:
                x = u / self.dt + (1.0 - PHYSICS["implicit_theta"]) * self._per_l(self.lin[v], u)
                if nk is not None:
                    x = x + 1.5 * nk - 0.5 * self.prev.get(k, nk)
                if self.bc_rows:
                    x = self._rows(x, self.t0 if k == "temp" else 0.0)
                x = self._solve(self.imp[v], x)
            out[k] = x
        self.prev = n
        return out


def _exact_steps(g, nr, k, dt, ekman, fields, scheme="cnab2", boundary=True):
    model = _ExactModel(g, nr, dt, ekman, scheme, bc_rows=scheme == "cnab2")
    if not boundary:
        model.t0 = 0.0
    s = {n: g.dense(a) for n, a in fields.items()}
    for _ in range(k):
        s = model.step(s)
    return s


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad() if kind != "gradient" else torch.enable_grad():
        if kind == "ensemble":
            cfgs = _members(case)
            # the order of the handles: members of one angular grid together, by first appearance
            slots = {}
            for i, c in enumerate(cfgs):
                slots.setdefault(c["lmax"], []).append(i)
            out = []
            for lmax, idx in slots.items():
                g = _exact_grid(lmax, cfgs[idx[0]]["nlat"], cfgs[idx[0]]["nlon"])
                parts = []
                for i in idx:
                    c = cfgs[i]
                    f = _state(seed * 64 + i, lmax, c["nr"], FIELDS[:5])
                    s = _exact_steps(g, c["nr"], case["k"], case["dt"], c["ekman"], f, boundary=False)
                    parts.append({n: g.packed(s[n]) for n in FIELDS[:5]})
                out.append([torch.cat([p[n] for p in parts], 1) for n in FIELDS[:5]])
            return out
        g = _exact_grid(case["lmax"], case["nlat"], case["nlon"])
        nr = case["nr"]
        if kind == "synth":
            gen = _generator(seed)
            return torch.stack([g.synth(g.dense(_random_field(gen, case["lmax"], nr, 1.0, 1.5, False)))
                                for _ in range(case["nfield"])])
        if kind == "roundtrip":
            gen = _generator(seed)
            T, S = (g.dense(_random_field(gen, case["lmax"], nr, 1.0, 1.5, True)) for _ in range(2))
            vt, vp = g.synth_vector(T, S)
            order = _modes(case["lmax"])[2]
            back = [g.packed(x)[:, :, torch.as_tensor(order, device="cuda")] for x in g.analysis_vector(vt, vp)]
            return [v.transpose(1, 2).contiguous() for v in (vt, vp)] + [p for b in back for p in (b[0], b[1])]
        if kind == "gradient":
            order = torch.as_tensor(_modes(case["lmax"])[2], device="cuda")
            f = _state(seed, case["lmax"], nr, FIELDS[:5])
            gen = _generator(seed + (1 << 40))
            lam = _random_field(gen, case["lmax"], nr, 1.0, 1.0, False)
            leaves = [f[n].requires_grad_() for n in ("temp", "u_tor", "u_pol")]
            s = _exact_steps(g, nr, case["k"], case["dt"], PHYSICS["ekman"], f)
            grads = torch.autograd.grad((g.packed(s["temp"]) * lam).sum(), leaves)
            return dict(gradient=tuple(tuple(x[c][:, order] for c in range(2)) for x in grads),
                        fields=[g.packed(s[n]).detach() for n in FIELDS[:5]])
        f = _state(seed, case["lmax"], nr, _names(case))
        s = _exact_steps(g, nr, case["k"], case["dt"], PHYSICS["ekman"], f, case["scheme"])
        return [g.packed(s[n]) for n in _names(case)]
