"""Performance cases of the MD step: what a user of the framework has it do.

Every case goes through the public C-ABI / Context / Batch calls the way an MD
program does: the context with its k-space tables, the start configuration and
the caller's own (pinned) host arrays exist before the pass; one pass is a
force evaluation, a number of steps called one by one with the field set
before each, or a segment of steps between two reads of the state, followed by
the read of the state into the caller's arrays.

kinds
  force   a configuration handed over, its force and energies read back (a
          relaxation, a structure comparison, a driver with its own integrator)
  calls   fg_set_uniform_E + fg_nose_poincare once per step, the energies of
          every step on the host (the reference's own call pattern)
  run     a Nose-Poincare segment of `steps` steps (fg_run_steps)
  film    an epitaxial film through part of its hysteresis loop, the field
          wave evaluated on the device (fg_set_wave)
  acou    leapfrog with the acoustic displacements as dynamic variables
  sites   a solid solution: its own Born charge and local field on every site
  sweep   the temperature points of a cooling sweep stepped as one batch

A segment is kept to 100 steps or fewer: the motion is chaotic, and longer ones
compare how two roundings have been amplified rather than two computations.

`prec` is the context's precision: "f64" (FP64 throughout) or "mixed" (FP32
fields and transforms; its callers keep the fields in FP32).  The parameters
are the BaTiO3 set of the reference's examples.
"""
import ctypes as C
import math

import numpy as np
import torch

import feram_b200 as fb
from feram_b200 import lib

# ---- BaTiO3 (the parameter set of the reference's example decks) ------------
A0, MASS, ACOU_MASS = 3.94, 39.0, 46.44
ZSTAR, EPS_INF = 9.956, 5.24
KAPPA2, ALPHA, GAMMA = 5.502, 110.4, -163.1
J = (-2.648, 3.894, 0.898, -0.789, 0.562, 0.358, 0.179)
B11, B12, B44 = 126.0, 44.9, 50.3
B1XX, B1YY, B4YZ = -211.0, -19.3, -7.75
GPA, DT = -5.0, 0.002
EPI_STRAIN, WAVE_PERIOD, E_AMP = -0.01, 400, 0.002
KELVIN_EV, ELEMENTARY, HARTREE_BOHR = 11604.45, 1.60217653, 14.399644


def _deck(c, L, kelvin):
    kind = c["kind"]
    film = kind == "film"
    t = ["method = '%s'" % ("lf" if kind == "acou" else "md"), "GPa = %r" % GPA, "kelvin = %r" % kelvin,
         "mass_amu = %r" % MASS, "bulk_or_film = '%s'" % ("epit" if film else "bulk"), "L = %d %d %d" % L,
         "a0 = %r" % A0, "dt = %r" % DT, "Q_Nose = %r" % _q_nose(L), "P_kappa2 = %r" % KAPPA2, "P_alpha = %r" % ALPHA,
         "P_gamma = %r" % GAMMA, "j = " + " ".join(repr(v) for v in J), "B11 = %r" % B11, "B12 = %r" % B12,
         "B44 = %r" % B44, "B1xx = %r" % B1XX, "B1yy = %r" % B1YY, "B4yz = %r" % B4YZ, "Z_star = %r" % ZSTAR,
         "epsilon_inf = %r" % EPS_INF, "external_E_field = 0.0 0.0 %r" % (E_AMP if film else 0.001)]
    if kind == "acou":
        t.append("acoustic_mass_amu = %r" % ACOU_MASS)
    if film:
        t += ["epi_strain = %r" % EPI_STRAIN, "E_wave_type = 'triangular_cos'", "n_E_wave_period = %d" % WAVE_PERIOD,
              "n_thermalize = 0", "n_average = 100000"]
    return "\n".join(t) + "\n"


def _q_nose(L):
    """The thermostat's mass grows with the number of sites (1 at 64^3)."""
    return max(0.1, L[0] * L[1] * L[2] / 64.0 ** 3)


def _supercells(c):
    """[(L, kelvin)] of a case: one, or the points of a sweep."""
    if c["kind"] != "sweep":
        return [((c["Lx"], c["Ly"], c["Lz"]), 300.0)]
    edges = [int(v) for v in c["edges"].split()]
    return [((n, n, n), 450.0 - 5.0 * i) for i, n in enumerate(edges)]


def _field(i):
    """The uniform field a `calls` program sets before step i (a slow ramp down)."""
    return [0.0, 0.0, 0.001 * (1.0 - 0.002 * (i + 1))]


def _start(c, L, kelvin, seed):
    """Start arrays (Lz, Ly, Lx, 3) of one supercell, FP32-representable in
    the mixed case: polarized dipoles and Maxwell-Boltzmann momenta."""
    rng = np.random.default_rng([seed, *L])
    n = (L[2], L[1], L[0])
    u = 0.09 + 0.04 * rng.standard_normal(n + (3,))
    p = math.sqrt(_mass(MASS) * kelvin / KELVIN_EV) * rng.standard_normal(n + (3,))
    f = {"u": u, "p": p}
    if c["kind"] == "acou":
        f["ar"] = 0.003 * rng.standard_normal(n + (3,))
        f["ap"] = math.sqrt(_mass(ACOU_MASS) * kelvin / KELVIN_EV) * rng.standard_normal(n + (3,))
    if c["kind"] == "sites":
        f["z"] = ZSTAR * (1.0 + 0.05 * rng.standard_normal(n + (1,)))
        f["e"] = 0.0005 * rng.standard_normal(n + (3,))
    if c["prec"] == "mixed":
        f = {k: v.astype(np.float32).astype(np.float64) for k, v in f.items()}
    return f


def _mass(amu):
    return amu / 9648.53377163899  # eV A^-2 ps^2


# ---- the cases ---------------------------------------------------------------
def _one(name, kind, L, prec, steps=0):
    return {"name": name, "kind": kind, "Lx": L[0], "Ly": L[1], "Lz": L[2], "prec": prec, "steps": steps}


def listed():
    return [
        # the smallest call: one force evaluation of a 16^3 cell (the reference's own example size)
        _one("force_16_f64", "force", (16, 16, 16), "f64"),
        # stepping a small cell from the host, one call per step: latency and launches
        _one("calls_16_f64", "calls", (16, 16, 16), "f64", 50),
        _one("calls_32_mixed", "calls", (32, 32, 32), "mixed", 50),
        # a force evaluation of a mid-size cell that is no power of two
        _one("force_60x50x36_mixed", "force", (60, 50, 36), "mixed"),
        # an ordinary production size, both precisions
        _one("run_64_f64", "run", (64, 64, 64), "f64", 100),
        _one("run_64_mixed", "run", (64, 64, 64), "mixed", 100),
        # a ragged cell (a domain-wall study: long in one direction)
        _one("run_96x40x90_mixed", "run", (96, 40, 90), "mixed", 100),
        # the benchmark's size
        _one("run_128_mixed", "run", (128, 128, 128), "mixed", 100),
        _one("run_128_f64", "run", (128, 128, 128), "f64", 100),
        # a thin film in its hysteresis loop
        _one("film_64x64x32_mixed", "film", (64, 64, 32), "mixed", 60),
        # acoustic MD
        _one("acou_48_f64", "acou", (48, 48, 48), "f64", 100),
        # the points of a cooling sweep, the sizes of a finite-size study
        {"name": "sweep_16_to_64_mixed", "kind": "sweep", "prec": "mixed", "steps": 60,
         "edges": "16 16 16 24 24 24 32 32 32 48 48 64"},
    ]



def _smooth(lo, hi, even):
    """Edges the transforms take: products of 2, 3 and 5 (Lx: an even one whose half is such a product)."""
    out = []
    for n in range(lo, hi + 1):
        m = n
        for q in (2, 3, 5):
            while m % q == 0:
                m //= q
        if m == 1 and not (even and n % 2):
            out.append(n)
    return out


def draw(rng):
    def edge(lo, hi, even=False):
        t = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return min(_smooth(lo, hi, even), key=lambda n: abs(n - t))

    kind = rng.choice(["force", "calls", "run", "run", "run", "film", "acou", "sites", "sweep"])
    prec = rng.choice(["f64", "mixed"])
    if kind == "sweep":
        edges = sorted(rng.choice([12, 16, 18, 20, 24, 32, 36, 40, 48, 64]) for _ in range(rng.randint(4, 10)))
        return {"kind": kind, "prec": prec, "steps": rng.randint(30, 60), "edges": " ".join(map(str, edges))}
    hi = {"force": 64, "calls": 64, "run": 128, "film": 96, "acou": 64, "sites": 48}[kind]
    if rng.random() < 0.4 and kind != "film":  # a cube
        n = edge(12, hi, True)
        L = (n, n, n)
    else:
        L = (edge(12, hi, True), edge(12, hi), edge(12, hi, kind == "film"))
    c = _one("", kind, L, prec, 0 if kind == "force" else rng.randint(20, 50) if kind == "calls" else rng.randint(30, 60))
    del c["name"]
    return c


# ---- preparation ---------------------------------------------------------------
class _Cell:
    """One supercell of a case: its context and the caller's host arrays."""


def _host_array(shape):
    """Pinned host array of the caller (numpy view kept alive by its tensor)."""
    return torch.zeros(shape, dtype=torch.float64, pin_memory=True)


def _padded(c, L, a):
    t = _host_array((L[2], L[1] + 1, 2 * (L[0] // 2 + 1), a.shape[-1]))
    t[:, :L[1], :L[0], :] = torch.from_numpy(a)
    return t


def _ptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_double))


def _ok(ctx, rc):
    if rc:
        raise RuntimeError("[%d] %s" % (rc, ctx.last_error()))


def _setup(c, cell, ctx, L, kelvin, seed):
    cell.ctx, cell.L = ctx, L
    cell.h = {k: _padded(c, L, v) for k, v in _start(c, L, kelvin, seed).items()}
    shape = cell.h["u"].shape
    keys = ("F",) if c["kind"] == "force" else ("u", "p", "ar", "ap") if c["kind"] == "acou" else ("u", "p")
    cell.out = {k: _host_array(shape) for k in keys}
    cell.f32 = {k: torch.zeros(shape, dtype=torch.float32) for k in cell.out} if c["prec"] == "mixed" else None
    cell.strain = np.zeros(6)
    cell.scal = [C.c_double(), C.c_double(), C.c_double()]
    cell.e = fb.fg_energy()
    ctx.build_tables()
    if c["kind"] == "sites":
        ctx.upload_site_arrays(Z_starR=cell.h["z"].numpy().copy(), E_field_local=cell.h["e"].numpy().copy())
    ctx.set_state(cell.h["u"].numpy(), cell.h["p"].numpy(), 1.0, 0.0, 0.0)
    if c["kind"] == "film":
        ctx.set_uniform_E([0.0, 0.0, E_AMP])
    elif c["kind"] != "sites":
        ctx.set_uniform_E([0.0, 0.0, 0.001])
    if c["kind"] == "force":
        return
    if c["kind"] == "acou":
        ctx.set_acou(cell.h["ar"].numpy(), cell.h["ap"].numpy())
        ctx.mirror_force_mirror()
        return
    # initialize_dipoR's tail and H0 as molecular_dynamics sets it
    e = ctx.mirror_force_mirror()
    e.dipo_kinetic = ctx.kinetic_energy_dipo()
    ctx.nose_poincare_hamiltonian(e)
    ctx.set_thermostat(1.0, 0.0, e.H_Nose_Poincare)
    if c["kind"] == "film":
        ctx.set_wave(True, 0)


def prepare(case, seed):
    c = case
    prec = fb.FG_PREC_MIXED if c["prec"] == "mixed" else fb.FG_PREC_FP64
    cells = _supercells(c)
    ps = [fb.params_from_text(_deck(c, L, kelvin)) for L, kelvin in cells]
    st = {"case": c, "cells": [], "step": 0, "batch": None}
    if c["kind"] == "sweep":
        st["batch"] = fb.Batch(ps, prec)
    for i, (L, kelvin) in enumerate(cells):
        cell = _Cell()
        _setup(c, cell, st["batch"][i] if st["batch"] else fb.Context(ps[i], prec), L, kelvin, seed + 1000003 * i)
        st["cells"].append(cell)
    return st


# ---- one pass --------------------------------------------------------------------
def _numbers(c, v):
    return np.array(v, dtype=np.float32 if c["prec"] == "mixed" else np.float64)


def _energies(e):
    return [getattr(e, n) for n, _ in e._fields_]


def _read(c, cell):
    """The state (of a force evaluation: the force) into the caller's arrays;
    FP32 ones for the mixed path."""
    ctx, o = cell.ctx, cell.out
    ptr = lambda k: _ptr(o[k]) if k in o else None  # noqa: E731
    _ok(ctx, lib().fg_get_state(ctx._h, ptr("u"), ptr("p"), ptr("F"),
                                cell.strain.ctypes.data_as(C.POINTER(C.c_double)), *[C.byref(v) for v in cell.scal]))
    if c["kind"] == "acou":
        _ok(ctx, lib().fg_get_acou(ctx._h, ptr("ar"), ptr("ap"), None))
    out = {k: o[k] if cell.f32 is None else cell.f32[k].copy_(o[k]) for k in o}
    out["strain"] = _numbers(c, cell.strain)
    if c["kind"] not in ("force", "acou"):
        out["thermostat"] = _numbers(c, [v.value for v in cell.scal[:2]])
    return out


def run(state):
    c, cells, n = state["case"], state["cells"], state["case"]["steps"]
    cell = cells[0]
    ctx = cell.ctx
    if c["kind"] == "force":
        _ok(ctx, lib().fg_set_state(ctx._h, _ptr(cell.h["u"]), None, 1.0, 0.0, 0.0))
        e = ctx.mirror_force_mirror(cell.e)
        out = _read(c, cell)
        out["energies"] = _numbers(c, _energies(e)[2:11])
        return out
    if c["kind"] == "calls":
        rows = []
        for i in range(state["step"], state["step"] + n):
            ctx.set_uniform_E(_field(i))
            rows.append(_energies(ctx.nose_poincare(cell.e)))
        state["step"] += n
        out = _read(c, cell)
        out["energies"] = _numbers(c, rows)
        return out
    if c["kind"] == "sweep":
        es = state["batch"].step(n)
        return {"cells": [dict(_read(c, x), energies=_numbers(c, _energies(e))) for x, e in zip(cells, es)]} \
            if len(cells) <= 9 else _merged(c, cells, es)
    e = ctx.run_steps(n, cell.e)
    out = _read(c, cell)
    out["energies"] = _numbers(c, _energies(e)[:11] if c["kind"] == "acou" else _energies(e))
    return out


def _merged(c, cells, es):
    """A long sweep's outputs: the fields per replica, the small arrays stacked."""
    outs = [_read(c, x) for x in cells]
    d = {"cells": [{k: o[k] for k in ("u", "p")} for o in outs]}
    for k in ("strain", "thermostat"):
        d[k] = np.stack([o[k] for o in outs])
    d["energies"] = _numbers(c, [_energies(e) for e in es])
    return d


# ---- the least work of a pass ------------------------------------------------------
def work(case):
    c = case
    w = 4 if c["prec"] == "mixed" else 8
    nc = 12 if c["kind"] in ("acou", "sites") else 9  # transformed components each way
    nf = 6 if c["kind"] == "acou" else 3              # displacement (and momentum) components
    by = fl = 0.0
    for L, _ in _supercells(c):
        n = L[0] * L[1] * L[2]
        # per site and step: u and p read and written, F written and read (the
        # next kick); each half spectrum (one real word per site) written and
        # read by the forward x-y / z split and again by the inverse one; the
        # dipole table's 6 words per half-spectrum point
        if c["kind"] == "force":
            by += n * (w * (3 + 3 + 4 * nc + 3) + 2 * 3 * 8)  # and the host arrays in and out
        else:
            by += n * (w * (4 * nf + 6 + 4 * nc + 3) * c["steps"] + 2 * nf * 8)
        # real transforms (2.5 n log2 n each, forward and inverse), the k-space
        # solve (about 300 per half-spectrum point), the site polynomial, the
        # strain couplings and the integrator (about 200 per site)
        fl += n * (2 * nc * 2.5 * math.log2(n) + 150 + 200) * max(1, c["steps"])
    return {"bytes": by, "flops": fl}


# ---- the same in 64 bits with torch -------------------------------------------------
class _Exact:
    """The effective Hamiltonian of one supercell in torch float64 (fields
    (3, z, y, x)), written from its equations: Fourier-space dipole-dipole and
    short-range interactions, on-site polynomial, strain relaxed exactly."""

    def __init__(self, c, L, kelvin):
        self.c, self.L, self.kelvin = c, L, kelvin
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.N = L[0] * L[1] * L[2]
        self.Q = _q_nose(L)
        self.dims = (1, 2, 3)
        self.film = c["kind"] == "film"
        self._k()
        self.S = self._short()
        self.Lr = self._long()
        H = np.zeros((6, 6))
        H[:3, :3] = B12
        H[range(3), range(3)] = B11
        H[range(3, 6), range(3, 6)] = B44
        self.H = H * self.N
        B = np.zeros((6, 6))
        B[:3, :3] = B1YY / 2
        B[range(3), range(3)] = B1XX / 2
        B[range(3, 6), range(3, 6)] = B4YZ
        self.HC2 = B
        self.pV = np.array([GPA * 0.01 / ELEMENTARY * self.N * A0 ** 3] * 3 + [0.0] * 3)
        self.Z, self.E = ZSTAR, torch.zeros(3, 1, 1, 1, dtype=torch.float64, device=self.dev)
        self.Eloc = 0.0

    def t(self, a):
        return torch.as_tensor(a, dtype=torch.float64, device=self.dev)

    def _k(self):
        def wrapped(n):
            k = np.arange(n) / n
            return np.where(k > 0.5, k - 1.0, k)
        x = self.t(np.arange(self.L[0] // 2 + 1) / self.L[0])
        y, z = self.t(wrapped(self.L[1])), self.t(wrapped(self.L[2]))
        self.kf = (x[None, None, :], y[None, :, None], z[:, None, None])
        self.k = tuple(v * (2 * math.pi / A0) for v in self.kf)

    def r2c(self, f):
        return torch.fft.rfftn(f, dim=tuple(range(f.dim() - 3, f.dim())))

    def c2r(self, K):
        """z and y complex, then x with the imaginary parts of its first and
        last bin dropped (the half-complex convention)."""
        d = K.dim()
        K = torch.fft.ifftn(K, dim=(d - 3, d - 2))
        K[..., 0].imag.zero_()
        K[..., -1].imag.zero_()
        return torch.fft.irfft(K, n=self.L[0], dim=-1)

    def _short(self):
        T = np.zeros((3, 3, self.L[2], self.L[1], self.L[0]))
        for a in range(3):
            T[a, a, 0, 0, 0] = 2 * KAPPA2
        for i in np.ndindex(3, 3, 3):
            d = tuple(v - 1 for v in i)
            shell = sum(v * v for v in d)
            for a in range(3):
                for b in range(3):
                    if shell == 1 and a == b:
                        v = J[0] if d[a] == 0 else J[1]
                    elif shell == 2:
                        v = (J[3] if d[a] == 0 else J[2]) if a == b else J[4] * d[a] * d[b]
                    elif shell == 3:
                        v = J[5] if a == b else J[6] * d[a] * d[b]
                    else:
                        continue
                    T[a, b, d[2], d[1], d[0]] = v
        return self.r2c(self.t(T)).real

    def _long(self):
        """Ewald sum of the dipole-dipole interaction per unit Z*^2."""
        L = self.L
        kap = math.sqrt(math.pi) / A0 / self.N ** (1.0 / 6)
        mx = [24 // n for n in L]
        r = [self.t(np.arange(n) * A0) for n in L]
        T = torch.zeros(3, 3, L[2], L[1], L[0], dtype=torch.float64, device=self.dev)
        for jz in range(-1 - mx[2], mx[2] + 1):
            for jy in range(-1 - mx[1], mx[1] + 1):
                for jx in range(-1 - mx[0], mx[0] + 1):
                    v = ((r[0] + jx * L[0] * A0)[None, None, :], (r[1] + jy * L[1] * A0)[None, :, None],
                         (r[2] + jz * L[2] * A0)[:, None, None])
                    rr = v[0] ** 2 + v[1] ** 2 + v[2] ** 2
                    if jx == jy == jz == 0:
                        rr[0, 0, 0] = 1e30
                    rn = rr.sqrt()
                    g = 2 / math.sqrt(math.pi) * kap * torch.exp(-kap * kap * rr)
                    ec = torch.erfc(kap * rn) / rn
                    Bd = (ec + g) / rr
                    Cd = (3 * ec / rr + g * (2 * kap * kap + 3 / rr)) / rr
                    for a in range(3):
                        T[a, a] += Bd
                        for b in range(3):
                            T[a, b] -= v[a] * v[b] * Cd
        for a in range(3):
            T[a, a, 0, 0, 0] -= 4 / math.sqrt(math.pi) * kap ** 3 / 3
        K = self.r2c(T).real
        for nz in range(-mx[2], mx[2] + 1):
            for ny in range(-mx[1], mx[1] + 1):
                for nx in range(-mx[0], mx[0] + 1):
                    G = tuple((self.kf[i] + n) * (2 * math.pi / A0) for i, n in enumerate((nx, ny, nz)))
                    gg = G[0] ** 2 + G[1] ** 2 + G[2] ** 2
                    if nx == ny == nz == 0:
                        gg[0, 0, 0] = 1e30
                    w = 4 * math.pi / A0 ** 3 * torch.exp(-gg / (4 * kap * kap)) / gg
                    for a in range(3):
                        for b in range(3):
                            K[a, b] += G[a] * G[b] * w
        return K * (HARTREE_BOHR / EPS_INF)

    def mirror(self, f):
        if self.film:
            h = self.L[2] // 2
            lo = f[:, :h].flip(1)
            f[0, h:], f[1, h:], f[2, h:] = -lo[0], -lo[1], lo[2]
        return f

    def coupling(self, w, u):
        return torch.stack([2 * w[0] * u[0] + w[4] * u[2] + w[5] * u[1], 2 * w[1] * u[1] + w[3] * u[2] + w[5] * u[0],
                            2 * w[2] * u[2] + w[3] * u[1] + w[4] * u[0]])

    def half(self, X):
        return float(X[..., 0].sum() / 2 + X[..., 1:-1].sum() + X[..., -1].sum() / 2)

    def force(self, u, ar=None):
        """Force on every site; the energies (short .. modulation) in self.e."""
        self.mirror(u)
        k1, k2, k3 = self.k
        Fs = self.c2r(torch.einsum("abzyx,bzyx->azyx", self.S + 0j, self.r2c(u)))
        Fl = self.Z * self.c2r(torch.einsum("abzyx,bzyx->azyx", self.Lr + 0j, self.r2c(self.Z * u)))
        F = Fs + Fl
        E = self.E + self.Eloc
        d = torch.stack([u[0] * u[0], u[1] * u[1], u[2] * u[2], u[1] * u[2], u[2] * u[0], u[0] * u[1]])
        uu = d[0] + d[1] + d[2]
        for a in range(3):
            F[a] += u[a] * ((4 * ALPHA + 2 * GAMMA) * uu - 2 * GAMMA * d[a])
        e = [float((u * Fs).sum()) / 2, float((u * Fl).sum()) / 2, -float((self.Z * u * E).sum()),
             float((ALPHA * uu * uu + GAMMA * (d[0] * d[1] + d[1] * d[2] + d[2] * d[0])).sum())]
        F -= self.Z * E
        # homogeneous strain
        h = self.HC2 @ d.sum(self.dims).cpu().numpy() + self.pV
        if self.film:
            st = np.array([EPI_STRAIN, EPI_STRAIN, (-2 * self.H[2, 0] * EPI_STRAIN - h[2]) / self.H[2, 2],
                           -h[3] / self.H[3, 3], -h[4] / self.H[4, 4], 0.0])
        else:
            st = -np.linalg.solve(self.H, h)
        self.strain = st
        e += [st @ self.H @ st / 2, st @ h]
        F += self.coupling(st @ self.HC2, u)
        # inhomogeneous strain
        D = self.r2c(d)
        hx, hy = B1XX / 2, B1YY / 2
        cs = torch.stack([k1 * (hx * D[0] + hy * (D[1] + D[2])) + B4YZ * (k3 * D[4] + k2 * D[5]),
                          k2 * (hx * D[1] + hy * (D[0] + D[2])) + B4YZ * (k3 * D[3] + k1 * D[5]),
                          k3 * (hx * D[2] + hy * (D[0] + D[1])) + B4YZ * (k2 * D[3] + k1 * D[4])])
        kk = [k + torch.zeros_like(D[0].real) for k in self.k]
        K = torch.stack([torch.stack([(B12 + B44) * kk[a] * kk[b] if a != b else
                                      (B11 - B44) * kk[a] * kk[a] + B44 * (kk[0] ** 2 + kk[1] ** 2 + kk[2] ** 2)
                                      for b in range(3)], -1) for a in range(3)], -2)
        if ar is None:
            K0 = K.clone()
            K0[0, 0, 0] = torch.eye(3, dtype=torch.float64, device=self.dev)
            A = torch.linalg.solve(K0 + 0j, -cs.movedim(0, -1).unsqueeze(-1)).squeeze(-1).movedim(-1, 0)
            A[:, 0, 0, 0] = 0
        else:
            A = 1j * self.r2c(ar)
        KA = torch.einsum("zyxab,bzyx->azyx", K + 0j, A)
        if ar is not None:
            self.da = self.c2r(-1j * (cs + KA))
        e += [self.half((A.conj() * KA).real.sum(0)) / self.N, self.half((A.conj() * cs).real.sum(0)) * 2 / self.N, 0.0]
        eta = self.c2r(torch.stack([k1 * A[0], k2 * A[1], k3 * A[2], k3 * A[1] + k2 * A[2], k1 * A[2] + k3 * A[0],
                                    k2 * A[0] + k1 * A[1]]))
        w = [hx * eta[0] + hy * (eta[1] + eta[2]), hx * eta[1] + hy * (eta[0] + eta[2]),
             hx * eta[2] + hy * (eta[0] + eta[1])] + [B4YZ * eta[i] for i in (3, 4, 5)]
        F += self.coupling(w, u)
        self.e = e
        return self.mirror(F)

    def kinetic(self, p, m):
        q = p[:, : self.L[2] // 2] if self.film else p
        return float((q * q).sum()) / m / 2 * (2 if self.film else 1)

    def hamiltonian(self):
        kT = self.kelvin / KELVIN_EV
        return (self.ke / self.s ** 2 + sum(self.e) + self.pi ** 2 / 2 / self.Q + 3 * self.N * kT * math.log(self.s) -
                self.H0) * self.s

    def np_start(self, u, p):
        self.s, self.pi, self.H0 = 1.0, 0.0, 0.0
        self.F = self.force(u)
        self.ke = self.kinetic(p, _mass(MASS))
        self.H0 = self.hamiltonian()

    def np_step(self, u, p):
        m, kT, h = _mass(MASS), self.kelvin / KELVIN_EV, DT / 2
        p -= h * self.s * self.F
        self.ke = self.kinetic(p, m)
        cb = 3 * self.N * kT * (1 + math.log(self.s)) - self.ke / self.s ** 2 + sum(self.e) - self.H0
        cb = h * cb - self.pi
        self.pi = -2 * cb / (1 + math.sqrt(1 - cb * DT / self.Q))
        a, s0 = h * self.pi / self.Q, self.s
        self.s = s0 * (1 + a) / (1 - a)
        u += h * (1 / self.s + 1 / s0) / m * p
        self.F = self.force(u)
        dH = self.hamiltonian() / self.s
        self.pi += h * (2 * self.ke / self.s ** 2 - 3 * self.N * kT) - h * dH
        p -= h * self.s * self.F
        self.ke = self.kinetic(p, m)

    def energies(self, acou=None):
        v = [acou or 0.0, self.ke] + self.e
        if acou is not None:
            return v
        return v + [self.ke / self.s ** 2 + sum(self.e), self.hamiltonian()]

    def wave(self, i):
        P = WAVE_PERIOD
        return E_AMP * (abs(i % P - P // 2) - P // 4) / (P / 4.0)

    def set_E(self, v):
        self.E = self.t(v).reshape(3, 1, 1, 1)


def _exact_cell(c, L, kelvin, seed):
    X = _Exact(c, L, kelvin)
    f = {k: X.t(v).movedim(-1, 0).contiguous() for k, v in _start(c, L, kelvin, seed).items()}
    u, p, n = f["u"], f["p"], c["steps"]
    X.set_E([0.0, 0.0, E_AMP if c["kind"] == "film" else 0.0 if c["kind"] == "sites" else 0.001])
    if c["kind"] == "sites":
        X.Z, X.Eloc = f["z"][0], f["e"]

    def padded(a):
        t = torch.zeros(L[2], L[1] + 1, 2 * (L[0] // 2 + 1), 3, dtype=torch.float64, device=a.device)
        t[:, :L[1], :L[0]] = a.movedim(0, -1)
        return t

    if c["kind"] == "force":
        F = X.force(u)
        return {"F": padded(F), "strain": X.strain, "energies": np.array(X.e)}
    if c["kind"] == "acou":
        m, ma = _mass(MASS), _mass(ACOU_MASS)
        ar, ap = f["ar"], f["ap"]
        for _ in range(n):
            u += DT / m * p
            ar += DT / ma * ap
            F = X.force(u, ar)
            p -= DT * F
            ap -= DT * X.da
        X.ke = X.kinetic(p, m)
        return {"u": padded(u), "p": padded(p), "ar": padded(ar), "ap": padded(ap), "strain": X.strain,
                "energies": np.array(X.energies(X.kinetic(ap, ma)))}
    X.np_start(u, p)
    rows = []
    for i in range(n):
        if c["kind"] == "calls":
            X.set_E(_field(i))
        elif c["kind"] == "film":
            X.set_E([0.0, 0.0, X.wave(i + 1)])
        X.np_step(u, p)
        if c["kind"] == "calls" or i == n - 1:
            rows.append(X.energies())
    return {"u": padded(u), "p": padded(p), "strain": X.strain, "thermostat": np.array([X.s, X.pi]),
            "energies": np.array(rows if c["kind"] == "calls" else rows[-1])}


def exact(case, seed):
    c = case
    outs = [_exact_cell(c, L, kelvin, seed + 1000003 * i) for i, (L, kelvin) in enumerate(_supercells(c))]
    if c["kind"] != "sweep":
        return outs[0]
    if len(outs) <= 9:
        return {"cells": outs}
    d = {"cells": [{k: o[k] for k in ("u", "p")} for o in outs]}
    for k in ("strain", "thermostat", "energies"):
        d[k] = np.stack([o[k] for o in outs])
    return d
