"""The work that users of this package have it do, as cases that can be timed.

Kinds of cases, each through the entry point that a user's program calls:

  step      one RK4 step of a closure of the serial solver
            (``RHSfunctions.advanceQ_RK4``), FP64 or FP32 fields; with
            ``stats`` the step is followed by ``computeAllStats``, as a run that
            records its energy and dissipation history does
  graph     the same step as one CUDA-graph replay (``StepGraph``)
  rhs       one right-hand-side evaluation (``main.computeRHS``): the RHS, the
            closure force and, where the model has one, its coefficient
  mhd       one RK4 step of the MPI solver's MHD (``mpi.advanceQ_RK4``), plain
            or with the t-model on both fields
  ensemble  one RK4 step of a set of independent runs of uneven sizes, one
            batch per grid size (``ensemble.Batch``)
  train     steps of the learned closure's training (``MLPModel.train``):
            forward, backward and Adam

Initial fields are random solenoidal fields with a filled spectrum (k^4 rise,
k^-5/3 range, exponential tail at the cutoff), or the Taylor-Green vortex,
made with torch from the seed.  ``exact`` restates each kind in 64 bits with
torch.fft.  The Kahan compensation array of FP32 runs is the rounding residue
of the stage sums; it is not an output.
"""
import math
import os

import numpy as np
import torch

from pyspectral_b200 import Classes as C
from pyspectral_b200 import RHSfunctions as R
from pyspectral_b200 import _capi, mpi
from pyspectral_b200.ensemble import Batch
from pyspectral_b200.learned import MLPModel

DEV = "cuda"
TWO_PI = 2.0 * math.pi
RK4 = (1.0 / 4, 1.0 / 3, 1.0 / 2, 1.0)
TURB = {"dns": 0, "smag": 1, "tmodel": 2, "stau": "Static tau-model", "dtau": "Dynamic tau-model",
        "dsmag": 7, "learned": "learned"}
MODEL = os.path.join(os.path.dirname(os.path.abspath(C.__file__)), "models", "sgs_mlp.npz")


def _c(name, kind, closure, n1, n2, n3, bits, **more):
    d = {"name": name, "kind": kind, "closure": closure, "n1": n1, "n2": n2, "n3": n3, "bits": bits}
    d.update(more)
    return d


def listed():
    return [
        # Taylor-Green validation run: 32^3 DNS in FP64, energy and dissipation
        # recorded after every step; the smallest call, launches and host latency count
        _c("tgv32_dns_f64", "step", "dns", 32, 32, 32, 64, init="tgv", nu=1.0 / 1600, dt=0.01, stats=True),
        # the headline LES: 64^3 with the learned closure in FP32, steps replayed from a graph
        _c("les64_learned_f32", "graph", "learned", 64, 64, 64, 32, nu=1e-3, dt=2e-3),
        # the plain FP64 path it is compared with
        _c("les64_smag_f64", "step", "smag", 64, 64, 64, 64, nu=1e-3, dt=2e-3),
        # a non-cubic grid with 108-, 72- and 162-point transforms: a caller's own RK loop around the RHS
        _c("ragged_smag_f32", "rhs", "smag", 72, 48, 108, 32, nu=1e-3, dt=2e-3),
        # dynamic tau-model RHS, the closure with the most work per evaluation
        _c("dtau64_f64", "rhs", "dtau", 64, 64, 64, 64, nu=1e-3, dt=2e-3),
        # decaying isotropic turbulence at 128^3: Smagorinsky and the t-model in FP64
        _c("hit128_smag_f64", "step", "smag", 128, 128, 128, 64, nu=1e-3, dt=2e-3),
        _c("hit128_tmodel_f64", "step", "tmodel", 128, 128, 128, 64, nu=1e-3, dt=1e-3),
        # MHD precision study: 128^3, t-model on both fields, FP32
        _c("mhd128_tmodel_f32", "mhd", "tmodel", 128, 128, 128, 32, nu=2e-3, dt=1e-3),
        # the learned closure at twice its training resolution
        _c("les128_learned_f32", "step", "learned", 128, 128, 128, 32, nu=1e-3, dt=2e-3),
        # the DNS that generates the learned closure's training data: the largest grid
        _c("dns256_f32", "step", "dns", 256, 256, 256, 32, nu=5e-4, dt=1e-3),
        # a sweep of decaying-turbulence runs: 8 each at 32^3, 48^3 (Smagorinsky) and 64^3 (learned)
        _c("ensemble24_f32", "ensemble", "smag+learned", 32, 48, 64, 32, nu=1e-3, dt=2e-3, runs=8),
        # training of the closure's network: minibatches of 16384 points, forward, backward, Adam
        _c("train_w32", "train", "relu", 16384, 32, 4, 32, nu=0.0, dt=2e-3),
    ]


# transform lengths N, 3N/2 and 2N that factor as 2^a 3^b
SIZES = (16, 24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        r = rng.random()
        n = rng.choice(SIZES)
        n1 = n2 = n3 = n
        if rng.random() < 0.35:  # non-cubic, the sides within a factor of about two
            near = [s for s in SIZES if n / 2 <= s <= 2 * n]
            n1, n2, n3 = rng.choice(near), rng.choice(near), rng.choice(near)
        bits = rng.choice((32, 64))
        nu = math.exp(rng.uniform(math.log(5e-4), math.log(5e-3)))
        dt = 0.1 / max(n1, n2, n3)
        if r < 0.62:
            closure = rng.choice(("dns", "smag", "smag", "learned", "tmodel", "stau"))
            c = _c("", rng.choice(("step", "graph")), closure, n1, n2, n3, bits, nu=nu, dt=dt,
                   stats=rng.random() < 0.2)
            if c["kind"] == "graph":
                c.pop("stats")
        elif r < 0.78:
            c = _c("", "rhs", rng.choice(("dns", "smag", "dsmag", "tmodel", "dtau")), n1, n2, n3, bits, nu=nu, dt=dt)
        elif r < 0.88:
            c = _c("", "mhd", rng.choice(("plain", "tmodel")), n1, n2, n3, bits, nu=nu, dt=dt)
        elif r < 0.95:
            a = rng.choice((16, 24, 32))
            c = _c("", "ensemble", "smag+learned", a, rng.choice((36, 48)), 64, 32, nu=nu, dt=2e-3,
                   runs=rng.randint(1, 12))
        else:
            c = _c("", "train", "relu", rng.choice((2048, 8192, 12000, 16384, 65536)), rng.choice((32, 64)),
                   rng.randint(1, 8), 32, nu=0.0, dt=2e-3)
        c.pop("name")
        if _cost(c) <= most:
            return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _wave(n1, n2, n3):
    k = [torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=torch.float64) for n in (n1, n2)]
    k1, k2 = k[0][:, None, None], k[1][None, :, None]
    k3 = torch.arange(n3 // 2 + 1, device=DEV, dtype=torch.float64)[None, None, :]
    return k1, k2, k3


def _solenoidal(n1, n2, n3, g):
    """Spectrum (3, n1, n2, n3//2+1) of a random solenoidal field of unit rms
    components, rfftn / sqrt(n1 n2 n3) as the serial solver's state; the
    Nyquist modes are zero."""
    k1, k2, k3 = _wave(n1, n2, n3)
    k = torch.sqrt(k1 * k1 + k2 * k2 + k3 * k3)
    kd = 0.5 * min(n1, n2, n3)
    amp = (k / 3.0) ** 2 / (1.0 + (k / 3.0) ** 2) ** (17.0 / 12.0) / (k + 1e-30) * torch.exp(-2.0 * k / kd)
    u = torch.randn((3, n1, n2, n3), generator=g, device=DEV, dtype=torch.float64)
    u = torch.fft.rfftn(u, dim=(1, 2, 3)) * amp
    div = (k1 * u[0] + k2 * u[1] + k3 * u[2]) / (k * k + 1e-50)
    u = torch.stack([u[0] - k1 * div, u[1] - k2 * div, u[2] - k3 * div])
    u[:, n1 // 2], u[:, :, n2 // 2], u[:, :, :, n3 // 2] = 0, 0, 0
    e = (u.abs() ** 2).sum() * 2 / (n1 * n2 * n3)
    return (u * torch.sqrt(3.0 * n1 * n2 * n3 / e)) / math.sqrt(n1 * n2 * n3)


def _tgv(n1, n2, n3, g):
    """Taylor-Green vortex at a random phase (the seed's)."""
    a = torch.rand(3, generator=g, device=DEV, dtype=torch.float64) * TWO_PI
    x, y, z = (torch.arange(n, device=DEV, dtype=torch.float64) * (TWO_PI / n) + a[i]
               for i, n in enumerate((n1, n2, n3)))
    x, y, z = x[:, None, None], y[None, :, None], z[None, None, :]
    u = torch.stack([torch.sin(x) * torch.cos(y) * torch.cos(z), -torch.cos(x) * torch.sin(y) * torch.cos(z),
                     torch.zeros((n1, n2, n3), device=DEV, dtype=torch.float64)])
    return torch.fft.rfftn(u, dim=(1, 2, 3)) / math.sqrt(n1 * n2 * n3)


def _cd(bits):
    return torch.complex128 if bits == 64 else torch.complex64


def _state0(c, seed):
    make = _tgv if c.get("init") == "tgv" else _solenoidal
    return make(c["n1"], c["n2"], c["n3"], _gen(seed)).to(_cd(c["bits"])).contiguous()


def _coords(n1, n2, n3):
    a = [np.arange(n) * (TWO_PI / n) for n in (n1, n2, n3)]
    sh = (n1, n2, n3)
    return (np.broadcast_to(a[0][:, None, None], sh), np.broadcast_to(a[1][None, :, None], sh),
            np.broadcast_to(a[2][None, None, :], sh))


def _physical6(c, seed):
    """Physical velocity and magnetic field, independent solenoidal fields."""
    n = (c["n1"], c["n2"], c["n3"])
    g = _gen(seed)
    s = torch.cat([_solenoidal(*n, g), _solenoidal(*n, g)])
    f = torch.fft.irfftn(s * math.sqrt(n[0] * n[1] * n[2]), s=n, dim=(1, 2, 3))
    return f.to(torch.float64 if c["bits"] == 64 else torch.float32)


def _ens_runs(c, seed):
    """[(N, closure, nu, state)] of an ensemble: viscosities log-uniform over a decade."""
    out = []
    g = _gen(seed)
    lognu = torch.rand(3 * c["runs"], generator=g, device=DEV, dtype=torch.float64).cpu().numpy()
    for s, N in enumerate((c["n1"], c["n2"], c["n3"])):
        for r in range(c["runs"]):
            nu = 5e-4 * 10.0 ** float(lognu[s * c["runs"] + r])
            out.append((N, "learned" if N == 64 else "smag", nu, _solenoidal(N, N, N, g).to(_cd(c["bits"]))))
    return out


def _samples(c, seed):
    """Features (velocity gradients and the filter width) and eddy-viscosity
    stresses with noise, four minibatches of points."""
    g = _gen(seed)
    n = 4 * c["n1"]
    G = torch.randn((n, 9), generator=g, device=DEV, dtype=torch.float32)
    X = torch.cat([G, torch.full((n, 1), TWO_PI / 64, device=DEV)], 1).contiguous()
    J = G.view(n, 3, 3)
    S = 0.5 * (J + J.transpose(1, 2))
    T = -0.02 * S.pow(2).sum((1, 2)).sqrt()[:, None, None] * S
    T = torch.stack([T[:, 0, 0], T[:, 1, 1], T[:, 2, 2], T[:, 0, 1], T[:, 0, 2], T[:, 1, 2]], 1)
    T = T + 0.005 * torch.randn(T.shape, generator=g, device=DEV)
    return X, T.contiguous()


def _fresh_params(c, seed):
    rs = np.random.RandomState(int(seed) & 0x7FFFFFFF)
    h = c["n2"]
    parts = []
    for fo, fi in ((h, 10), (h, h), (6, h)):
        b = 1.0 / math.sqrt(fi)
        parts += [rs.uniform(-b, b, size=fo * fi), np.zeros(fo)]
    return np.concatenate(parts).astype(np.float32)


T0, CT = 0.5, 0.1       # time and coefficient of the t-models
TAU_A, TAU_B = 0.02, 0.01  # static tau-model


def prepare(case, seed):
    c = case
    n = (c["n1"], c["n2"], c["n3"])
    k = c["kind"]
    if k in ("step", "graph", "rhs"):
        q = _state0(c, seed)
        grid = C.gridclass(*n, *_coords(*n), min(n) // 2)
        model = MLPModel.load(MODEL) if c["closure"] == "learned" else None
        tau = {"dt0": TAU_A, "dt1": TAU_B} if c["closure"] == "stau" else {}
        main = C.variables(0, TURB[c["closure"]], 0, 0, 0, 0, grid, q[0], q[1], q[2], T0, c["dt"], c["nu"], Ct=CT,
                           precision=c["bits"], model=model, les_delta=TWO_PI / 64 if model else None, **tau)
        s = {"kind": k, "main": main, "grid": grid, "stats": c.get("stats", False), "q": q,
             "util": C.utilitiesClass(), "closure": c["closure"]}
        if k == "graph":
            s["graph"] = R.StepGraph(main, grid, 1)
        return s
    if k == "mhd":
        f = _physical6(c, seed)
        grid = mpi.gridclass(*n, *_coords(*n), min(n) // 2)
        main = mpi.variables("MHD", 0, 0, 0, 0, grid, *f, t=T0, dt=c["dt"], nu=c["nu"], precision=c["bits"],
                             closure="tmodel" if c["closure"] == "tmodel" else None, Ct=CT)
        return {"kind": k, "main": main, "grid": grid}
    if k == "ensemble":
        model = MLPModel.load(MODEL)
        runs = _ens_runs(c, seed)
        batches, states = [], []
        for N in n:
            mine = [r for r in runs if r[0] == N]
            learned = mine[0][1] == "learned"
            b = Batch(_capi.Context(N, N, N, precision=c["bits"]), _capi.LEARNED if learned else _capi.SMAG, len(mine))
            for i, (_, _, nu, st) in enumerate(mine):
                st = st.contiguous()
                p = _capi.make_params(nu=nu, dt=c["dt"], mlp_params=model.params.data_ptr() if learned else None,
                                      mlp_norm=model.norm.data_ptr() if learned else None, les_delta=TWO_PI / N,
                                      mlp_act=model.act if learned else 0, mlp_hidden=model.hidden if learned else 0)
                b.set_run(i, st, torch.zeros_like(st) if c["bits"] == 32 else None, p)
                states.append(st)
            batches.append(b)
        return {"kind": k, "batches": batches, "states": states, "model": model}
    X, T = _samples(c, seed)
    model = MLPModel(params=_fresh_params(c, seed), act=c["closure"], hidden=c["n2"])
    model.fit_norm(X, T)
    return {"kind": k, "model": model, "X": X, "T": T, "ctx": _capi.Context(32, 32, 32, precision=32),
            "steps": c["n3"], "batch": c["n1"], "lr": c["dt"]}


def run(state):
    s = state
    k = s["kind"]
    if k == "step":
        main, grid = s["main"], s["grid"]
        R.advanceQ_RK4(main, grid, None, s["util"])
        out = [main.Q, main.U]
        return out + [list(s["util"].computeAllStats(main, grid))] if s["stats"] else out
    if k == "graph":
        s["graph"].replay()
        return [s["main"].Q, s["main"].U]
    if k == "rhs":
        main = s["main"]
        main.Q = s["q"]
        main.computeRHS(main, s["grid"], None, s["util"])
        out = [main.Q, main.U]
        if main.W0 is not None:
            out.append(main.W0)
        if s["closure"] == "dtau":
            out.append(main.tau)
        if s["closure"] == "dsmag":
            out.append(main.Cs_sqr)
        return out
    if k == "mhd":
        mpi.advanceQ_RK4(s["main"], s["grid"])
        return [s["main"].Q, s["main"].U]
    if k == "ensemble":
        for b in s["batches"]:
            b.step(1)
        return s["states"]
    m = s["model"]
    m.train(s["ctx"], s["X"], s["T"], s["steps"], batch=s["batch"], lr=s["lr"])
    return [m.params, m.m, m.v]


# ---------------------------------------------------------------------------
# algorithmic work
# ---------------------------------------------------------------------------
def _fft3(n, M, Kz, fin, fout):
    """Operations of fin inverse and fout forward padded 3-D real transforms,
    only the lines that carry data: 5 M log2 M per complex line."""
    (n1, n2, _), (m1, m2, m3) = n, M

    def line(m):
        return 5.0 * m * math.log2(m)
    per = n2 * Kz * line(m1) + m1 * Kz * line(m2) + 0.5 * m1 * m2 * line(m3)
    return (fin + fout) * per


def _rhs_flops(closure, n):
    n1, n2, n3 = n
    M = tuple(3 * a // 2 for a in n)
    F = tuple(2 * a for a in n)
    m3, f3 = M[0] * M[1] * M[2], F[0] * F[1] * F[2]
    spec = n1 * n2 * (n3 // 2 + 1)
    if closure == "dns":
        return _fft3(n, M, n3 // 2, 3, 6) + 6.0 * m3 + 120.0 * spec
    if closure == "smag":
        return _fft3(n, M, n3 // 2, 9, 12) + 40.0 * m3 + 200.0 * spec
    if closure == "dsmag":
        return 2 * _fft3(n, M, n3 // 2, 9, 12) + 80.0 * m3 + 600.0 * spec
    if closure == "learned":
        return _fft3(n, M, n3 // 2, 12, 6) + (12.0 + 2.0 * (10 * 32 + 32 * 32 + 32 * 6)) * m3 + 120.0 * spec
    # memory models: products of u on the 2x grid (its spectrum kept whole), products of u with the unresolved part
    pl = _fft3(n, F, n3 // 2, 3, 0) + _fft3(F, F, n3, 3, 6) + 120.0 * F[0] * F[1] * n3
    plql = _fft3(n, F, n3 // 2, 0, 6) + 18.0 * f3 + 120.0 * spec
    return (pl + plql) * (2 if closure == "dtau" else 1)


def _cost(c):
    return work(c)["flops"]


def work(case):
    c = case
    n = (c["n1"], c["n2"], c["n3"])
    e = 16.0 if c["bits"] == 64 else 8.0
    k = c["kind"]
    spec = n[0] * n[1] * (n[2] // 2 + 1)
    if k in ("step", "graph"):
        # state read and written, the state as read by the last stage written;
        # FP32 runs also read and write the compensation
        fields = 9 + (6 if c["bits"] == 32 else 0) + (3 if c.get("stats") else 0)
        return {"bytes": e * spec * fields, "flops": 4 * (_rhs_flops(c["closure"], n) + 30.0 * spec)}
    if k == "rhs":
        return {"bytes": e * spec * (9 if c["closure"] == "dns" else 12), "flops": _rhs_flops(c["closure"], n)}
    if k == "mhd":
        kz = int((n[2] // 2) * 2.0 / 3.0)
        f = _fft3(n, n, kz, 6, 9) + 20.0 * n[0] * n[1] * n[2] + 200.0 * spec
        if c["closure"] == "tmodel":
            F = tuple(2 * a for a in n)
            f3 = F[0] * F[1] * F[2]
            f += _fft3(n, F, kz, 6, 9) + _fft3(F, F, n[2], 6, 9) + 60.0 * f3 + 200.0 * F[0] * F[1] * n[2]
        fields = 21 + (12 if c["bits"] == 32 else 0)  # state in and out, read state, forcing
        return {"bytes": e * spec * fields, "flops": 4 * (f + 60.0 * spec)}
    if k == "ensemble":
        b = fl = 0.0
        for N in n:
            s = N * N * (N // 2 + 1)
            b += c["runs"] * e * s * 12
            fl += c["runs"] * 4 * (_rhs_flops("learned" if N == 64 else "smag", (N, N, N)) + 30.0 * s)
        return {"bytes": b, "flops": fl}
    h, pts = c["n2"], float(c["n1"]) * c["n3"]
    npar = h * h + 18 * h + 6
    # forward and two products per weight backward; points read once, Adam's parameters and moments
    return {"bytes": pts * 4.0 * 17 + c["n3"] * 7.0 * 4.0 * npar,
            "flops": pts * 6.0 * (10 * h + h * h + 6 * h) + c["n3"] * 12.0 * npar}


# ---------------------------------------------------------------------------
# the same in 64 bits with torch
# ---------------------------------------------------------------------------
def _rows(n, m, drop):
    """(source rows, padded rows) of an axis of n points embedded in m points;
    drop: without the N/2 row."""
    i = torch.arange(n, device=DEV)
    if drop:
        i = i[i != n // 2]
    return i, torch.where(i < n // 2, i, i + (m - n))


class _X:
    """A grid's transforms and wavenumbers in 64 bits."""

    def __init__(self, n, M, drop):
        self.n, self.M, self.h = n, M, n[2] // 2
        self.r = [_rows(n[a], M[a], drop) for a in (0, 1)]
        self.N = n[0] * n[1] * n[2]
        self.k = _wave(*n)
        k1, k2, k3 = self.k
        # the N/2 rows are the -N/2 modes, as fftfreq has them
        self.ks = k1 * k1 + k2 * k2 + k3 * k3 + 1e-50

    def up(self, x):
        (a, A), (b, B) = self.r
        out = torch.zeros(self.M[:2] + (self.M[2] // 2 + 1,), dtype=torch.complex128, device=DEV)
        out[A[:, None], B[None, :], :self.h] = x[a[:, None], b[None, :], :self.h]
        return out

    def down(self, X):
        (a, A), (b, B) = self.r
        out = torch.zeros(self.n[:2] + (self.h + 1,), dtype=torch.complex128, device=DEV)
        out[a[:, None], b[None, :], :self.h] = X[A[:, None], B[None, :], :self.h]
        return out

    def phys(self, X):
        return torch.fft.irfftn(X, s=self.M)

    def spec(self, x):
        return torch.fft.rfftn(x)


def _press(k, ks, P):
    k1, k2, k3 = k
    return -(k1 * k1 * P[0] + k2 * k2 * P[1] + k3 * k3 * P[2] + 2 * k1 * k2 * P[3] + 2 * k1 * k3 * P[4]
             + 2 * k2 * k3 * P[5]) / ks


def _diverge(k, P):
    k1, k2, k3 = k
    return [-1j * (k1 * P[0] + k2 * P[3] + k3 * P[4]), -1j * (k1 * P[3] + k2 * P[1] + k3 * P[5]),
            -1j * (k1 * P[4] + k2 * P[5] + k3 * P[2])]


def _advect(k, ks, nu, P, u):
    ph = _press(k, ks, P)
    return torch.stack([d - 1j * k[i] * ph - nu * ks * u[i] for i, d in enumerate(_diverge(k, P))])


PAIRS = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))


def _nyq0(q):
    q = q.clone()
    q[:, q.shape[1] // 2], q[:, :, q.shape[2] // 2], q[:, :, :, -1] = 0, 0, 0
    return q


def _strain_hat(k, u):
    k1, k2, k3 = k
    return [1j * k1 * u[0], 1j * k2 * u[1], 1j * k3 * u[2], 0.5j * (k2 * u[0] + k1 * u[1]),
            0.5j * (k3 * u[0] + k1 * u[2]), 0.5j * (k3 * u[1] + k2 * u[2])]


def _contract(S, T):
    return S[0] * T[0] + S[1] * T[1] + S[2] * T[2] + 2 * (S[3] * T[3] + S[4] * T[4] + S[5] * T[5])


def _sgs_force(k, ks, t):
    # the projection term is 1j k_i (1j k_m k_j tau_jm / k^2)
    proj = -1j * _press(k, ks, t)
    return torch.stack([d + 1j * k[i] * proj for i, d in enumerate(_diverge(k, t))])


def _mlp(X):
    d = np.load(MODEL)
    P = torch.as_tensor(d["params"].astype(np.float64), device=DEV)
    nr = torch.as_tensor(d["norm"].astype(np.float64), device=DEV)
    return _net(P, nr, X)


def _net(P, nr, X):
    h = int(round(-9 + math.sqrt(81 + P.numel() - 6)))
    o = 0
    W = []
    for fo, fi in ((h, 10), (h, h), (6, h)):
        W.append((P[o:o + fo * fi].view(fo, fi), P[o + fo * fi:o + fo * fi + fo]))
        o += fo * fi + fo
    x = (X - nr[:10]) * nr[10:20]
    for i, (w, b) in enumerate(W):
        x = x @ w.T + b
        if i < 2:
            x = torch.relu(x)
    return x * nr[26:32] + nr[20:26]


def _rhs32(closure, n, q, nu, delta):
    """RHS of the 3/2-padded closures: (rhs, state as read, closure force, coefficient)."""
    x = _X(n, tuple(3 * a // 2 for a in n), True)
    s = math.sqrt(1.5 ** 3 * math.sqrt(x.N))
    u = q if closure in ("smag", "dsmag") else _nyq0(q)
    w0 = cs2 = None
    ur = [x.phys(x.up(a)) * s for a in u]
    if closure == "learned":
        g = [x.phys(x.up(1j * x.k[j] * u[i])) * (s * s) for i in range(3) for j in range(3)]
        X = torch.stack([a.reshape(-1) for a in g] + [torch.full((ur[0].numel(),), delta, device=DEV,
                                                                 dtype=torch.float64)], 1)
        del g
        t = torch.cat([_mlp(b) for b in X.split(1 << 20)])
        del X
        P = [x.down(x.spec(ur[a] * ur[b] + t[:, m].reshape(ur[0].shape) / (s * s))) for m, (a, b) in enumerate(PAIRS)]
    else:
        P = [x.down(x.spec(ur[a] * ur[b])) for a, b in PAIRS]
    r = _advect(x.k, x.ks, nu, P, u)
    D = TWO_PI / (x.N ** (1.0 / 3.0))
    if closure in ("smag", "dsmag"):
        S = [x.phys(x.up(a)) * s for a in _strain_hat(x.k, u)]
        sm = torch.sqrt(2 * _contract(S, S))
        t = [x.down(x.spec(sm * a)) for a in S]
        if closure == "smag":
            cs2 = (0.16 ** 2)
        else:
            cs2 = _dsmag_cs2(x, s, u, ur, S, sm, D, min(n) // 2)
        w0 = _sgs_force(x.k, x.ks, [-2 * cs2 * D * D * a for a in t])
        r = r + w0
    return r, u, w0, cs2


def _box(n, kc):
    """The sharp test filter along one axis: |k| < kc."""
    m = torch.zeros(n, dtype=torch.float64, device=DEV)
    m[:kc] = 1
    m[n - kc + 1:] = 1
    return m


def _dsmag_cs2(x, s, u, ur, S, sm, D, kc):
    kt = int(kc / 2.0)
    f = _box(x.n[0], kt)[:, None, None] * _box(x.n[1], kt)[None, :, None]
    f3 = torch.zeros(x.h + 1, dtype=torch.float64, device=DEV)
    f3[:kt] = 1
    f = f * f3[None, None, :]
    uf = f * u
    vf = [x.phys(x.up(a)) * s for a in uf]
    Sf = [x.phys(x.up(a)) * s for a in _strain_hat(x.k, uf)]
    sf = torch.sqrt(2 * _contract(Sf, Sf))

    def back(a):
        return x.phys(x.up(a))
    L = [back(f * x.down(x.spec(ur[a] * ur[b])) - x.down(x.spec(vf[a] * vf[b]))) for a, b in PAIRS]
    M = [back(-2 * D * D * (4 * x.down(x.spec(sf * Sf[m])) - f * x.down(x.spec(sm * S[m])))) for m in range(6)]
    num = sum(L[m] * M[m] for m in range(6))
    den = sum(M[m] * M[m] for m in range(6))
    return num.mean() / den.mean()


def _memory(closure, n, q, nu):
    """RHS of the t-model and the tau-models on the 2x grid."""
    x = _X(n, tuple(2 * a for a in n), False)
    X = _X(x.M, x.M, False)
    s = math.sqrt(8.0 * math.sqrt(x.N))
    u = _nyq0(q)
    n1, n2, n3 = n

    def inside(i, N):
        return (i < N // 2) | (i > 2 * N - N // 2)
    i1, i2 = torch.arange(2 * n1, device=DEV), torch.arange(2 * n2, device=DEV)
    i3 = torch.arange(n3 + 1, device=DEV)
    res = inside(i1, n1)[:, None, None] & inside(i2, n2)[None, :, None] & (i3 < n3 // 2)[None, None, :]

    def stage(u, res):
        up = [x.up(a) for a in u]
        ur = [x.phys(a) * s for a in up]
        P = [X.spec(ur[a] * ur[b]) for a, b in PAIRS]
        PL = _advect(X.k, X.ks, nu, P, up)
        qr = [x.phys(torch.where(res, torch.zeros_like(a), a)) * s for a in PL]
        A = [x.down(x.spec(ur[a] * qr[b] + ur[b] * qr[a])) for a, b in PAIRS]
        d = _diverge(x.k, A)
        ph = _press(x.k, x.ks, A)
        Q = torch.stack([d[i] - 1j * x.k[i] * ph for i in range(3)])
        plain = _diverge(X.k, P)
        php = _press(X.k, X.ks, P)
        lead = [plain[i] + 1j * X.k[i] * php for i in range(3)]
        return torch.stack([x.down(a) for a in PL]), Q, lead

    PL, Q, lead = stage(u, res)
    if closure == "tmodel":
        tau = CT * T0
    elif closure == "stau":
        tau = TAU_A + TAU_B * T0
    else:
        kf = int((min(n) // 2) * 2.0 / 3.0)
        f = [(a.abs() < kf).to(torch.float64) for a in x.k]
        F = [(a.abs() < kf).to(torch.float64) for a in X.k]
        G, G2 = f[0] * f[1] * f[2], F[0] * F[1] * F[2]
        uf = G * u

        def low(i, N):
            return (i < kf) | (i >= 2 * N - kf + 1)
        resf = low(i1, n1)[:, None, None] & low(i2, n2)[None, :, None] & (i3 < kf)[None, None, :]
        _, Qf, leadf = stage(uf, resf)

        def dot(a, b):
            h = n3 // 2
            return (a[..., 1:h] * b[..., 1:h].conj()).sum() * 2 + (a[..., 0] * b[..., 0].conj()).sum()
        LE = sum(dot(G2 * (lead[i] - leadf[i]), x.up(uf[i])) for i in range(3)) / x.N
        a = sum(dot(G * Qf[i], uf[i]) for i in range(3)) / x.N
        b = sum(dot(Q[i], uf[i]) for i in range(3)) / x.N
        tau = float((LE.abs() / (a.abs() - b.abs() + 1e-5)).item())
    w0 = max(0.0, tau) * Q
    return PL + w0, u, w0, tau


def _rhs(c, n, q, nu, closure, delta):
    if closure in ("tmodel", "stau", "dtau"):
        return _memory(closure, n, q, nu)
    return _rhs32(closure, n, q, nu, delta)


def _rk4(q, dt, f):
    q0 = q
    u = None
    for a in RK4:
        r, u = f(q)
        q = q0 + dt * a * r
    return q, u


def _mhd_nl(k, ks, P):
    k1, k2, k3 = k
    ph = _press(k, ks, P)
    d = _diverge(k, P)
    return torch.stack([d[i] - 1j * k[i] * ph for i in range(3)] +
                       [1j * (k2 * P[8] - k3 * P[7]), 1j * (k3 * P[6] - k1 * P[8]), 1j * (k1 * P[7] - k2 * P[6])])


def _mhd_rhs(c, n, q, nu, force):
    x = _X(n, n, False)
    D = 1.0
    for a in (0, 1):
        D = D * (x.k[a].abs() < (n[a] // 2) * 2.0 / 3.0).to(torch.float64)
    m3 = torch.ones(n[2] // 2 + 1, dtype=torch.float64, device=DEV)
    m3[int((n[2] // 2) * 2.0 / 3.0):] = 0
    D = D * m3[None, None, :]
    st = D * q

    def prods(f):
        u, v, w, a, b, d = f
        return [u * u - a * a, v * v - b * b, w * w - d * d, u * v - a * b, u * w - a * d, v * w - b * d,
                v * d - w * b, w * a - u * d, u * b - v * a]
    P = [x.spec(a) for a in prods([x.phys(a) for a in st])]
    r = _mhd_nl(x.k, x.ks, P) - nu * x.ks * st
    r[:3] += force
    r = D * r
    if c["closure"] == "tmodel":
        F = tuple(2 * a for a in n)
        y, Y = _X(n, F, False), _X(F, F, False)
        DF = y.up(D + 0j).real

        def ph(X):
            return Y.phys(X) * 8.0

        def sp(a):
            return Y.spec(a) / 8.0
        f = [ph(y.up(a)) for a in st]
        QL = (1 - DF) * _mhd_nl(Y.k, Y.ks, [sp(a) for a in prods(f)])
        g = [ph(a) for a in QL]
        del QL
        # bilinear products about the state in the direction of its unresolved rate of change
        lin = [p - m for p, m in zip(prods([a + 0.5 * b for a, b in zip(f, g)]),
                                     prods([a - 0.5 * b for a, b in zip(f, g)]))]
        mem = _mhd_nl(x.k, x.ks, [y.down(sp(a)) for a in lin])
        r = r + (CT * T0) * D * mem
    return r, st


def exact(case, seed):
    c = case
    n = (c["n1"], c["n2"], c["n3"])
    k = c["kind"]
    if k in ("step", "graph"):
        q = _state0(c, seed).to(torch.complex128)
        q, u = _rk4(q, c["dt"], lambda v: _rhs(c, n, v, c["nu"], c["closure"], TWO_PI / 64)[:2])
        out = [q, u]
        if c.get("stats"):
            k1, k2, k3 = _wave(*n)
            h = n[2] // 2

            def dot(a):
                e = a.abs() ** 2
                return float((2 * e[..., 1:h].sum() + e[..., 0].sum()).item()) / (n[0] * n[1] * n[2])
            om = torch.stack([k2 * u[2] - k3 * u[1], k3 * u[0] - k1 * u[2], k1 * u[1] - k2 * u[0]])
            en, ens = 0.5 * dot(u), 0.5 * dot(om)
            eps = 2 * ens * c["nu"]
            out.append([ens, en, eps, (c["nu"] ** 3 / eps) ** 0.25, (c["nu"] / eps) ** 0.5,
                        en * math.sqrt(20.0 / (3.0 * c["nu"] * eps))])
        return out
    if k == "rhs":
        r, u, w0, coef = _rhs(c, n, _state0(c, seed).to(torch.complex128), c["nu"], c["closure"], TWO_PI / 64)
        out = [r, u]
        if w0 is not None:
            out.append(w0)
        if c["closure"] in ("dtau", "dsmag"):
            out.append(float(coef))
        return out
    if k == "mhd":
        q = torch.fft.rfftn(_physical6(c, seed).double(), dim=(1, 2, 3))
        x, y, z = (torch.as_tensor(np.ascontiguousarray(a), device=DEV) for a in _coords(*n))
        f = 0.25 * torch.stack([torch.sin(2 * x) * torch.cos(2 * y) * torch.cos(2 * z),
                                -torch.cos(2 * x) * torch.sin(2 * y) * torch.cos(2 * z), torch.zeros_like(x)])
        f = torch.fft.rfftn(f, dim=(1, 2, 3))
        return list(_rk4(q, c["dt"], lambda v: _mhd_rhs(c, n, v, c["nu"], f)))
    if k == "ensemble":
        out = []
        for N, closure, nu, st in _ens_runs(c, seed):
            out.append(_rk4(st.to(torch.complex128), c["dt"],
                            lambda v: _rhs(c, (N, N, N), v, nu, closure, TWO_PI / N)[:2])[0])
        return out
    # training: Adam on minibatches of one epoch's permutation, cosine learning rate
    X, T = (a.double() for a in _samples(c, seed))
    # the normalisation as prepare() leaves it, in 32 bits
    Xf, Tf = _samples(c, seed)
    nr = torch.cat([Xf.mean(0), 1.0 / Xf.std(0).clamp_min(1e-12), Tf.mean(0), Tf.std(0).clamp_min(1e-12)]).double()
    P = torch.as_tensor(_fresh_params(c, seed).astype(np.float64), device=DEV)
    m, v = torch.zeros_like(P), torch.zeros_like(P)
    g = torch.Generator(device=DEV)
    g.manual_seed(0)
    B, steps, pos = c["n1"], c["n3"], 0
    perm = torch.randperm(X.shape[0], generator=g, device=DEV)
    for s in range(steps):
        if pos + B > X.shape[0]:
            perm, pos = torch.randperm(X.shape[0], generator=g, device=DEV), 0
        i = perm[pos:pos + B].long()
        pos += B
        p = P.clone().requires_grad_(True)
        Y = (_net(p, nr, X[i]) - nr[20:26]) / nr[26:32]
        ((Y - (T[i] - nr[20:26]) / nr[26:32]) ** 2).mean().backward()
        m = 0.9 * m + 0.1 * p.grad
        v = 0.999 * v + 0.001 * p.grad ** 2
        lr = 1e-4 + 0.5 * (c["dt"] - 1e-4) * (1 + math.cos(math.pi * s / max(1, steps)))
        P = P - lr * (m / (1 - 0.9 ** (s + 1))) / (torch.sqrt(v / (1 - 0.999 ** (s + 1))) + 1e-8)
    return [P, m, v]
