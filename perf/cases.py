"""The work this framework does for its users, as cases that can be timed.

A case is one call sequence of a user's program through the public entry
points, on a grid and a batch of its own:

  single      c_primal, the tangents and the adjoint of one trajectory on host
              arrays (the reference package's own use)
  segments    c_batch_forward_dev + c_batch_adjoint_dev: the shadowing sweep
              over independent segments resident on the GPU
  gradient    c_primal + c_adjoint_exact_grad: one checkpoint interval of a
              differentiated trajectory, forward and backward
  uneven      c_multi_forward + c_multi_adjoint: instances with grids, Re and
              dt of their own
  kkt         one matrix-vector product of the least-squares-shadowing system
  spec2phys   the physical velocity field of one coefficient array

The library keeps one grid and its working sets per process, as the
reference does; that grid is the handle a program keeps, and it is set up
again only when a case of another grid is prepared.
"""
import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "shadow-channel_gb300"))
from channel import c_channel as cc  # noqa: E402
from channel import lss  # noqa: E402

DEV = "cuda" if torch.cuda.is_available() else "cpu"
FLUX = 2.0
UNEVEN_GRIDS = ((16, 33, 16), (32, 65, 32), (48, 97, 48))


def _case(name, kind, nx, ny, nz, steps, **more):
    c = dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, steps=steps, lx=2 * math.pi, lz=math.pi, re=3300.0, dt=0.005,
             segs=1, ntan=1, strength=1.0)
    c.update(more)
    return c


def listed():
    return [
        # the smallest call there is: one field for a plot or a probe
        _case("spec2phys-16", "spec2phys", 16, 33, 16, 1, re=2000.0, dt=0.01),
        # the reference's default grid: the drivers' tests and small studies, launch latency counts
        _case("single-16", "single", 16, 33, 16, 10, re=2000.0, dt=0.01),
        # one segment as the drivers run it: primal, two homogeneous tangents and a forced one, adjoint
        _case("single-32", "single", 32, 65, 32, 5, ntan=3),
        # a checkpoint interval of a differentiated time mean (dJ/dC0, dJ/dmeanU, dJ/dRe)
        _case("gradient-32", "gradient", 32, 65, 32, 10),
        # a shadowing system's product, the body of every MINRES iteration
        _case("kkt-16", "kkt", 16, 33, 16, 5, segs=8, re=2000.0, dt=0.01),
        # a small ensemble on the default grid
        _case("segments-16x12", "segments", 16, 33, 16, 8, segs=12, ntan=2, re=2000.0, dt=0.01),
        # an ensemble on a ragged grid: odd transform lengths, no size a power of two
        _case("segments-ragged", "segments", 28, 43, 18, 4, segs=5, ntan=2),
        # the headline workload: 64 segments, primal + 3 tangents + coupled adjoint
        _case("segments-32x64", "segments", 32, 65, 32, 3, segs=64, ntan=3),
        # a few segments of a finer grid
        _case("segments-48x4", "segments", 48, 97, 48, 2, segs=4, ntan=2),
        # a parameter study over grids, Reynolds numbers and time steps
        _case("uneven-24", "uneven", 48, 97, 48, 3, segs=24, ntan=1),
        # one segment between the small grids and the largest
        _case("single-64", "single", 64, 65, 64, 2),
        # the largest grid: forward and uncoupled adjoint of one checkpoint interval's steps
        _case("single-128", "single", 128, 129, 128, 1, lx=4 * math.pi, lz=2 * math.pi, dt=0.002, ntan=0, strength=0.0),
    ]


def draw(rng):
    def size(lo, hi, step):  # spread over the logarithm, transform lengths that factor into 2, 3, 5, 7
        while True:
            n = step * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)
            m = n // 2
            for f in (2, 3, 5, 7):
                while m % f == 0:
                    m //= f
            if m == 1 and lo <= n <= hi:
                return n

    kind = rng.choice(("single", "single", "segments", "segments", "segments", "gradient", "uneven", "kkt", "spec2phys"))
    while True:
        nx, nz = size(12, 128, 4), size(10, 128, 2)
        ny = 2 * round(math.exp(rng.uniform(math.log(17), math.log(129))) / 2) + 1
        segs = 1 if kind in ("single", "gradient", "spec2phys") else round(math.exp(rng.uniform(math.log(2), math.log(64))))
        steps = rng.randint(2, 10)
        ntan = rng.randint(1, 3)
        points = nx * ny * nz * segs * steps * (2 + ntan)
        if kind == "uneven":
            nx, ny, nz = UNEVEN_GRIDS[-1]
            segs, steps, ntan = rng.randint(3, 40), rng.randint(2, 4), 1
            points = 0
        if nx * ny * nz <= 500_000 and points <= 25_000_000:
            break
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=steps, lx=2 * math.pi, lz=math.pi,
                re=rng.uniform(2000.0, 4000.0), dt=rng.choice((0.002, 0.004, 0.005)), segs=segs, ntan=ntan,
                strength=rng.choice((0.0, 0.5, 1.0)))


# ---------------------------------------------------------------------------
# the handle: the library's grid, batch or operator
# ---------------------------------------------------------------------------

_held = {"key": None}


def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


def _instances(case):
    """(Nx, Ny, Nz, Re, dt) of each instance of an uneven batch."""
    rng = np.random.default_rng([case["segs"], int(case["re"])])
    pick = rng.integers(0, len(UNEVEN_GRIDS), case["segs"])
    return [UNEVEN_GRIDS[g] + (float(rng.uniform(2000.0, 4000.0)), float(rng.uniform(0.002, 0.005))) for g in pick]


def _inhomo(case):
    """Every tangent homogeneous but the last, which is mean-flux forced and coupled."""
    return [0] * (case["ntan"] - 1) + [1]


def _ints(v):
    return (ctypes.c_int * len(v))(*v)


def _doubles(v):
    return (ctypes.c_double * len(v))(*v)


def _hold(case):
    if _held["key"] == _key(case):
        return _held
    if _held["key"] is not None:
        cc.lib.c_batch_destroy()
        cc.lib.c_multi_destroy()
        cc.c_destroy()
    _held.clear()
    _held["key"] = None
    kind = case["kind"]
    if kind == "uneven":
        inst = _instances(case)
        n = len(inst)
        col = list(zip(*inst))
        rc = cc.lib.c_multi_init(n, _ints(col[0]), _ints(col[1]), _ints(col[2]), _doubles([case["lx"]] * n),
                                 _doubles([case["lz"]] * n), _doubles(col[3]), _doubles([FLUX] * n), _doubles(col[4]),
                                 case["steps"], case["ntan"], case["ntan"] - 1)
        assert rc == 0, cc.c_last_error_message()
    else:
        nsteps = case["segs"] * case["steps"] if kind == "kkt" else case["steps"]
        rc = cc.c_init(case["nx"], case["ny"], case["nz"], case["lx"], case["lz"], case["re"], FLUX, case["dt"], nsteps)
        assert rc == 0, cc.c_last_error_message()
    if kind == "segments":
        assert cc.lib.c_batch_init_steps(case["segs"], case["ntan"], case["ntan"] - 1, case["steps"]) == 0, \
            cc.c_last_error_message()
    if kind == "kkt":
        _held["starts"] = _window_starts(case)
        _held["kkt"] = lss.KKT(_held["starts"], case["steps"])
    if kind in ("segments", "kkt"):
        _held["stream"] = torch.cuda.ExternalStream(cc.lib.c_stream())
    _held["key"] = _key(case)
    return _held


def _window_seed(case):
    return _states(case["nx"], case["ny"], case["nz"], 1, 90125, True)[0]


def _window_starts(case):
    """The states at the window starts of one trajectory (the operator's own data, the same for every input)."""
    C = _window_seed(case).cpu().numpy()
    cc.c_primal(0, C)
    return np.stack([cc.c_getsoln(i * case["steps"]).copy() for i in range(case["segs"])])


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _states(nx, ny, nz, n, seed, laminar, amp=1e-2):
    """n seeded coefficient arrays [n][Nz][2][Ny-2][Nx/2] on the GPU: a full spectrum of complex normal noise that
    decays with every wave number and the Legendre index, as a developed field's does, on the laminar profile or
    (tangents, adjoints) without it; Hermitian on kx = 0, a real mean line, no kz = Nz/2 line."""
    R, D, X = ny - 2, ny - 4, nx // 2
    gen = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + nx * 101 + ny * 13 + nz)
    C = torch.randn((n, nz, 2, R, X, 2), dtype=torch.float64, device=DEV, generator=gen)
    C = torch.view_as_complex(C)
    kz = torch.arange(nz, device=DEV)
    kz = torch.minimum(kz, nz - kz).double()
    decay = (torch.exp(-kz / 3)[:, None, None, None] * torch.exp(-torch.arange(R, device=DEV).double() / 4)[None, None, :, None] *
             torch.exp(-torch.arange(X, device=DEV).double() / 3)[None, None, None, :])
    C = C * (amp * decay)
    C[:, 1:, 0, D:] = 0
    C[:, 0, 0, D:, 1:] = 0
    C[:, nz // 2] = 0
    for z in range(1, nz // 2):
        C[:, nz - z, :, :, 0] = torch.conj(C[:, z, :, :, 0])
    C[:, 0, :, :, 0] = C[:, 0, :, :, 0].real.to(C.dtype)
    if laminar:
        C[:, 0, 0, 0, 0] += 0.75 * FLUX
    return C.contiguous()


def _inputs(case, seed):
    """The initial states, tangents and adjoints (or the operand) of one pass, complex, on the GPU."""
    grid = (case["nx"], case["ny"], case["nz"])
    n, nt = case["segs"], max(case["ntan"], 0)
    if case["kind"] == "uneven":
        parts = {"C": [], "IC": [], "AC": []}
        for i, (nx, ny, nz, _, _) in enumerate(_instances(case)):
            parts["C"].append(_states(nx, ny, nz, 1, 64 * seed + i, True))
            parts["IC"].append(_states(nx, ny, nz, nt, 64 * seed + i + 20_000_003, False))
            parts["AC"].append(_states(nx, ny, nz, 1, 64 * seed + i + 40_000_003, False))
        return {k: [x for x in v] for k, v in parts.items()}
    if case["kind"] == "kkt":
        return {"x": _states(*grid, 2 * n - 1, seed, False)}
    d = {"C": _states(*grid, n, seed, True)}
    if case["kind"] in ("single", "segments"):
        if nt:
            d["IC"] = _states(*grid, n * nt, seed + 20_000_003, False)
        d["AC"] = _states(*grid, n, seed + 40_000_003, False)
    if case["kind"] == "gradient":
        d["AC"] = _states(*grid, 1, seed + 40_000_003, False)
        d["src"] = torch.zeros_like(d["AC"])  # the time mean's source: weights on the mean line
        d["src"][0, 0, 0, :, 0] = torch.randn(case["ny"] - 2, dtype=torch.float64, device=DEV,
                                              generator=torch.Generator(device=DEV).manual_seed(seed)) / case["steps"]
    return d


def prepare(case, seed):
    _hold(case)
    inp = _inputs(case, seed)
    s = {"case": dict(case)}
    kind = case["kind"]
    if kind == "segments":
        s["in"] = [inp["C"], inp["IC"], inp["AC"]]
        s["work"] = [torch.empty_like(x) for x in s["in"]]
        s["inhomo"] = _ints(_inhomo(case))
    elif kind == "kkt":
        s["x"] = torch.view_as_real(inp["x"]).reshape(-1).contiguous()
    elif kind == "uneven":
        s["in"] = [np.concatenate([x.cpu().numpy().ravel() for x in inp[k]]) for k in ("C", "IC", "AC")]
        s["work"] = [np.empty_like(x) for x in s["in"]]
        s["inhomo"] = _ints(_inhomo(case))
    else:
        s["in"] = {k: [x.cpu().numpy() for x in v] for k, v in inp.items()}
        s["work"] = {k: [np.empty_like(x) for x in v] for k, v in s["in"].items()}
        if kind == "spec2phys":
            s["flow"] = np.zeros((3, 3 * case["nx"] // 2, 3 * case["ny"] // 2, 3 * case["nz"] // 2))
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    case = state["case"]
    held = _hold(case)
    kind, n = case["kind"], case["steps"]
    if kind == "segments":
        C, IC, AC = state["work"]
        with torch.cuda.stream(held["stream"]):  # the sweeps update their arrays in place: start from the inputs
            for w, x in zip(state["work"], state["in"]):
                w.copy_(x)
        assert cc.lib.c_batch_forward_dev(0, n, C.data_ptr(), IC.data_ptr(), state["inhomo"]) == 0, \
            cc.c_last_error_message()
        assert cc.lib.c_batch_adjoint_dev(n, 0, AC.data_ptr(), case["strength"]) == 0, cc.c_last_error_message()
        return [torch.view_as_real(x) for x in (C, IC, AC)]
    if kind == "kkt":
        y = held["kkt"].matvec(state["x"])
        return [y, held["kkt"].zeta]
    if kind == "uneven":
        for w, x in zip(state["work"], state["in"]):
            w[...] = x
        C, IC, AC = state["work"]
        assert cc.lib.c_multi_forward(0, n, C.ctypes.data, IC.ctypes.data, state["inhomo"]) == 0, \
            cc.c_last_error_message()
        assert cc.lib.c_multi_adjoint(n, 0, AC.ctypes.data, case["strength"]) == 0, cc.c_last_error_message()
        return [C, IC, AC]
    work = state["work"]
    for k, v in state["in"].items():
        for w, x in zip(work[k], v):
            w[...] = x
    C = work["C"][0]
    if kind == "spec2phys":
        cc.c_spec2phys(C, state["flow"])
        return [state["flow"]]
    cc.c_primal(0, C)
    AC = work["AC"][0]
    if kind == "gradient":
        return [C, AC, *cc.c_adjoint_exact_grad(n, 0, AC, work["src"][0])]
    if case["ntan"]:
        for ic, inhomo in zip(work["IC"], _inhomo(case)):
            cc.c_tangent(0, n, ic, inhomo)
    cc.c_adjoint(n, 0, AC, 0, case["strength"])
    return [C, *work.get("IC", []), AC]


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------

def _grid_work(nx, ny, nz):
    """(coefficient bytes, nominal FP64 flop of one field's quadratures, of one plane transform over all planes)"""
    X, Q, R, D, pz, px = nx // 2, 3 * ny // 2, ny - 2, ny - 4, 3 * nz // 2, 3 * nx // 2
    quad = 4.0 * Q * (5 * D + 3 * R) * nz * X
    plane = Q * (X * 5 * pz * math.log2(pz) + pz * 2.5 * px * math.log2(px))
    return 16.0 * nz * 2 * R * X, quad, plane


def work(case):
    """Bytes: the arrays in and out and the stored trajectories; flop: three substages a step of the Legendre
    contractions and 9 plane transforms a forward field, 15 for the adjoint, 9 for the exact one."""
    kind, n, nt = case["kind"], case["steps"], case["ntan"]
    if kind == "uneven":
        grids = [i[:3] for i in _instances(case)]
    else:
        grids = [(case["nx"], case["ny"], case["nz"])] * case["segs"]
    nbytes = flops = 0.0
    for g in grids:
        cb, quad, plane = _grid_work(*g)
        fwd, adj = 3 * n * (quad + 9 * plane), 3 * n * (1.5 * quad + 15 * plane)
        if kind == "spec2phys":
            nbytes += cb + 8.0 * 3 * (3 * g[0] // 2) * (3 * g[1] // 2) * (3 * g[2] // 2)
            flops += quad * 0.5 + 3 * plane
        elif kind == "gradient":
            nbytes += cb * (5 + 3 * n)
            flops += fwd + 3 * n * (quad + 9 * plane)
        elif kind == "kkt":
            nbytes += cb * (4 + 3 * n)
            flops += fwd + adj
        else:
            nbytes += cb * (2 * (2 + nt) + (2 if nt else 1) * 3 * n)
            flops += (1 + nt) * fwd + adj
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same outputs from the equations: dense Legendre-Galerkin matrices,
# torch's FFT and solves, in 64 bits
# ---------------------------------------------------------------------------

class _Channel:
    """Semi-implicit RK3 steps of the channel in wall-normal velocity and vorticity form: u = (u, v, w) from
    alpha (v in the basis (1 - y^2)^2 P_n) and beta (vorticity in (1 - y^2) P_n)."""

    A, B = (1 / 3, -1 / 2, 1 / 3), (1 / 6, 2 / 3, 0.0)
    C, D = (1 / 2, 1 / 3, 1.0), (0.0, -1 / 6, -2 / 3)
    AA, AB = (1 / 3, -1 / 2, 1 / 3), (2 / 3, 1 / 6, 0.0)
    AC, AD = (1.0, 1 / 3, 1 / 2), (0.0, -2 / 3, -1 / 6)

    def __init__(self, nx, ny, nz, lx, lz, re, dt, flux=FLUX):
        dev = DEV
        self.nx, self.nz, self.X, self.q, self.R, self.Dq = nx, nz, nx // 2, 3 * ny // 2, ny - 2, ny - 4
        self.px, self.pz, self.dt, self.flux, self.nu = 3 * nx // 2, 3 * nz // 2, dt, flux, 1.0 / re
        y, w = np.polynomial.legendre.leggauss(self.q)
        eye, leg = np.eye(self.R), np.polynomial.legendre
        c1, c2 = leg.poly2leg([1, 0, -1]), leg.poly2leg([1, 0, -2, 0, 1])

        def basis(c, n, der):
            return np.stack([leg.legval(y, leg.legder(leg.legmul(c, eye[j]), der)) for j in range(n)], 1)

        q = [basis(c2, self.Dq, d) for d in (0, 1, 2)]
        r = [basis(c1, self.R, d) for d in (0, 1)]

        def t(a):
            return torch.tensor(a, dtype=torch.float64, device=dev)

        self.w = t(w)
        self.Q, self.Qp, self.Qpp = map(t, q)
        self.Rb, self.Rp = map(t, r)
        self.Qw, self.Qpw, self.Qppw = (t((x * w[:, None]).T.copy()) for x in q)
        self.Rw, self.Rpw = (t((x * w[:, None]).T.copy()) for x in r)
        self.Qs, self.Qps, self.Qpps = self.Qw @ self.Q, self.Qpw @ self.Qp, self.Qppw @ self.Qpp
        self.Rs, self.Rps = self.Rw @ self.Rb, self.Rpw @ self.Rp
        kz = np.fft.fftfreq(nz, 1.0 / nz) * (2 * math.pi / lz)
        kx = np.arange(self.X) * (2 * math.pi / lx)
        self.kz, self.kx = t(kz)[:, None, None], t(kx)[None, None, :]
        k2 = t(kz)[:, None] ** 2 + t(kx)[None, :] ** 2
        self.k2 = k2[:, None, :]
        self.k2n = self.k2.clone()
        self.k2n[0, 0, 0] = 1.0  # the mean mode goes by its own rule
        keep = torch.ones((nz, self.X), dtype=torch.float64, device=dev)
        keep[nz // 2] = 0
        self.keep = keep[:, None, :]
        mean = torch.zeros((nz, self.X), dtype=torch.float64, device=dev)
        mean[0, 0] = 1
        self.mean = mean[:, None, :]
        self.rows = [z for z in range(nz) if z != nz // 2]
        self.prow = [z if z < nz // 2 else z + nz // 2 for z in self.rows]
        self.lu = {}

    # -- fields ---------------------------------------------------------
    @staticmethod
    def mul(M, c):  # real matrix times complex columns [..., n, x]
        return torch.complex(M @ c.real, M @ c.imag)

    def velocity(self, c):
        """u, v, w, du/dy, dw/dy of coefficients [Nz][2][R][X], each [Nz][q][X]."""
        al, be = c[:, 0, :self.Dq], c[:, 1]
        v, p, d = self.mul(self.Q, al), self.mul(-self.Qp, al), self.mul(self.Qpp, al)
        g, e = self.mul(self.Rb, be), self.mul(self.Rp, be)
        kx, kz, k2 = self.kx, self.kz, self.k2n
        u, w = -1j * (kx * p + kz * g) / k2, 1j * (kx * g - kz * p) / k2
        du, dw = 1j * (kx * d - kz * e) / k2, 1j * (kx * e + kz * d) / k2
        a0 = c[0, 0, :, 0]
        b0 = c[0, 1, :, 0]

        def mean(x, col):
            return x * (1 - self.mean) + self.mean * col[None, :, None]

        full = self.mul
        return (mean(u, full(self.Rb, a0[:, None])[:, 0]), mean(v, torch.zeros_like(v[0, :, 0])),
                mean(w, full(self.Rb, b0[:, None])[:, 0]), mean(du, full(self.Rp, a0[:, None])[:, 0]),
                mean(dw, full(self.Rp, b0[:, None])[:, 0]))

    def physical(self, f):
        """[n][Nz][q][X] modes to [n][pz][q][px] values."""
        F = torch.zeros((f.shape[0], self.pz) + f.shape[2:3] + (self.px // 2 + 1,), dtype=f.dtype, device=f.device)
        F[:, self.prow, :, :self.X] = f[:, self.rows]
        F = torch.fft.ifft(F, dim=1) * self.pz
        F = torch.cat([F[..., :1].real.to(F.dtype), F[..., 1:]], -1)
        return torch.fft.irfft(F, n=self.px, dim=-1) * self.px

    def modes(self, p):
        """The kept modes [n][Nz][q][X] of values [n][pz][q][px]."""
        F = torch.fft.fft(torch.fft.rfft(p, dim=-1)[..., :self.X], dim=1) / (self.px * self.pz)
        out = torch.zeros((p.shape[0], self.nz) + p.shape[2:3] + (self.X,), dtype=F.dtype, device=F.device)
        out[:, self.rows] = F[:, self.prow]
        return out

    def fields(self, c):
        """Velocity and vorticity values, [6][pz][q][px]."""
        u, v, w, du, dw = self.velocity(c)
        ox, oz = dw - 1j * self.kz * v, -du + 1j * self.kx * v
        oy = 1j * self.kz * u - 1j * self.kx * w
        return self.physical(torch.stack([u, v, w, ox, oy, oz]))

    @staticmethod
    def cross(a, b):
        return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])

    # -- implicit solve -------------------------------------------------
    def bands(self, coef):
        """The alpha and beta operators M + nu coef dt D of every mode, and the mean line's."""
        k2 = self.k2n.reshape(-1)[:, None, None]
        h = self.nu * coef * self.dt
        a = -(k2 * self.Qs + self.Qps) + h * (k2 * k2 * self.Qs + 2 * k2 * self.Qps + self.Qpps)
        b = self.Rs - h * (self.Rps + k2 * self.Rs)
        return a, b, self.Rs - h * self.Rps

    def apply(self, M, c):  # [modes][n][n] times [Nz][n][X]
        x = c.permute(0, 2, 1).reshape(-1, c.shape[1])
        x = torch.view_as_real(x)
        return torch.view_as_complex((M @ x).contiguous()).reshape(self.nz, self.X, -1).permute(0, 2, 1)

    def solve(self, M, c, key=None):
        x = torch.view_as_real(c.permute(0, 2, 1).reshape(-1, c.shape[1]).contiguous())
        if key is None:
            x = torch.linalg.solve(M, x)
        else:
            if key not in self.lu:
                self.lu[key] = torch.linalg.lu_factor(M)
            x = torch.linalg.lu_solve(*self.lu[key], x)
        return torch.view_as_complex(x.contiguous()).reshape(self.nz, self.X, -1).permute(0, 2, 1)

    def rhs(self, h, adj=None):
        """Weighted quadratures of the nonlinear terms h = (x, y, z) (adj: S_x, S_z too): alpha, beta, mean lines."""
        kx, kz = self.kx, self.kz
        fa = self.mul(self.Qpw, 1j * (kx * h[0] + kz * h[2])) - self.k2 * self.mul(self.Qw, h[1])
        fb = self.mul(self.Rw, 1j * (kz * h[0] - kx * h[2]))
        f0, g0 = self.Rw @ h[0][0, :, 0].real, self.Rw @ h[2][0, :, 0].real
        if adj is not None:
            sx, sz = adj
            fa = fa + self.mul(self.Qppw, 1j * (kx * sz - kz * sx))
            fb = fb + self.mul(self.Rpw, 1j * (kz * sz + kx * sx))
            f0 = f0 + self.Rpw @ sz[0, :, 0].real
            g0 = g0 - self.Rpw @ sx[0, :, 0].real
        return fa, fb, f0, g0

    def substage(self, k, c, f, fnext, target, adjoint=False, cached=True):
        """Solves one substage of the carried right-hand side c with terms f; returns (solved state, next carried
        right-hand side).  target: the mean flux the solved mean line is corrected to."""
        a, b, cc_, d = (self.AA, self.AB, self.AC, self.AD) if adjoint else (self.A, self.B, self.C, self.D)
        dt, Dq = self.dt, self.Dq
        al, be = c[:, 0], c[:, 1]
        m0, m1 = al[0, :, 0], be[0, :, 0]
        if k == 0:
            Ma, Mb, M0 = self.bands(a[0])
            ea, eb = self.apply(Ma, al[:, :Dq]), self.apply(Mb, be)
            m0, m1 = self.mul(M0, m0[:, None])[:, 0], self.mul(M0, m1[:, None])[:, 0]
        else:
            ea, eb = al[:, :Dq], be
        La, Lb, L0 = self.bands(-b[k])
        xa = self.solve(La, (ea + dt * cc_[k] * f[0]), ("a", adjoint, k) if cached else None) * self.keep
        xb = self.solve(Lb, (eb + dt * cc_[k] * f[1]), ("b", adjoint, k) if cached else None) * self.keep
        one = self.Rw.sum(1)
        add = torch.linalg.solve(L0 if adjoint else self.Rs, one)

        def mean_solve(x):
            return torch.complex(torch.linalg.solve(L0, x.real), torch.linalg.solve(L0, x.imag))

        x0, x1 = mean_solve(m0 + dt * cc_[k] * f[2]), mean_solve(m1 + dt * cc_[k] * f[3])
        x0 = x0 + (target - (one * x0.real).sum()) * 0.5 * add
        rest = al[:, Dq:] * self.keep

        def pack(pa, pb, p0, p1):
            top = torch.cat([pa, rest], 1)
            top = top * (1 - self.mean) + self.mean * p0[None, :, None]
            bot = pb * (1 - self.mean) + self.mean * p1[None, :, None]
            return torch.stack([top, bot], 1)

        s = pack(xa, xb, x0, x1)
        if k == 2:
            return s, s
        g = f if fnext is None else fnext
        Ma, Mb, M0 = self.bands(a[k + 1])
        na = (self.apply(Ma, xa) + dt * d[k + 1] * g[0]) * self.keep
        nb = (self.apply(Mb, xb) + dt * d[k + 1] * g[1]) * self.keep
        n0 = self.mul(M0, x0[:, None])[:, 0] + dt * d[k + 1] * g[2]
        n1 = self.mul(M0, x1[:, None])[:, 0] + dt * d[k + 1] * g[3]
        return s, pack(na, nb, n0, n1)

    # -- sweeps ---------------------------------------------------------
    def primal(self, c, steps, cached=True, flux=None):
        """The states at every substage, [3 steps + 1]."""
        out, s = [c], c
        flux = self.flux if flux is None else flux
        for _ in range(steps):
            for k in range(3):
                p = self.fields(s)
                s, c = self.substage(k, c, self.rhs(self.modes(self.cross(p[:3], p[3:]))), None, flux, cached=cached)
                out.append(s)
        return out

    def tangent(self, traj, c, start, end, forced):
        out, s = {3 * start: c}, c
        for n in range(start, end):
            for k in range(3):
                p, t = self.fields(traj[3 * n + k]), self.fields(s)
                h = self.modes(self.cross(p[:3], t[3:]) + self.cross(t[:3], p[3:]))
                s, c = self.substage(k, c, self.rhs(h), None, 2.0 if forced else 0.0)
                out[3 * n + k + 1] = s
        return s, out

    def velocity_values(self, c):
        return self.physical(torch.stack(self.velocity(c)[:3]))

    def ddt_project(self, traj, i, v):
        hi, lo = (3, 0) if i == 0 else (3 * i, 3 * (i - 1))
        d = (traj[hi] - traj[lo]) / self.dt
        a, b, w = self.velocity_values(d), self.velocity_values(v), self.w[None, None, :, None]
        r = (a * b * w).sum() / (a * a * w).sum()
        return v - r * d, r

    def adjoint_terms(self, x, au):
        p = self.fields(x)
        S, T = self.modes(self.cross(p[:3], au)), self.modes(self.cross(au, p[3:]))
        kx, kz = self.kx, self.kz
        h = (-T[0] + 1j * kz * S[1], -T[1] - 1j * kz * S[0] + 1j * kx * S[2], -T[2] - 1j * kx * S[1])
        return self.rhs(h, (S[0], S[2]))

    def adjoint(self, traj, itraj, c, start, end, strength):
        s = c
        for n in range(start, end, -1):
            if strength:
                c = c - 0.5 * strength * self.dt * self.ddt_project(traj, n, itraj[3 * n])[0]
            for k in range(3):
                m = 3 * n - k - 1
                au = self.velocity_values(s)
                f = self.adjoint_terms(traj[m], au)
                g = self.adjoint_terms(traj[m - 1], au) if k < 2 else f
                s, c = self.substage(k, c, f, g, 0.0, adjoint=True)
            if strength:
                c = c - 0.5 * strength * self.dt * self.ddt_project(traj, n - 1, itraj[3 * (n - 1)])[0]
        return c


def _real(x):
    return torch.view_as_real(x.contiguous()).cpu()


def _exact_sweep(ch, C, ICs, AC, steps, forced, strength):
    traj = ch.primal(C, steps)
    ends, last = [], None
    for ic, f in zip(ICs, forced):
        e, last = ch.tangent(traj, ic, 0, steps, f)
        ends.append(e)
    return traj[-1], ends, ch.adjoint(traj, last, AC, steps, 0, strength)


def _exact_kkt(ch, x, windows, steps, start):
    traj = ch.primal(start, windows * steps)
    v, w = list(x[:windows]), list(x[windows:]) + [torch.zeros_like(x[0])]
    rv, rw, zeta = [], [], []
    for i in range(windows):
        a, b = i * steps, (i + 1) * steps
        end, itraj = ch.tangent(traj, ch.ddt_project(traj, a, v[i])[0], a, b, False)
        end, eta = ch.ddt_project(traj, b, end)
        zeta.append(-float(eta))
        back = ch.adjoint(traj, itraj, ch.ddt_project(traj, b, w[i])[0], b, a, 1.0)
        back = ch.ddt_project(traj, a, back)[0]
        rv.append((w[i - 1] if i else 0) - back)
        if i < windows - 1:
            rw.append(v[i + 1] - end)
    return [_real(torch.stack(rv + rw)).reshape(-1), np.array(zeta)]


def exact(case, seed):
    kind, n = case["kind"], case["steps"]
    fwd = work(case)["flops"]
    if fwd > 1e11:  # over about 20 s: no value
        return None
    inp = _inputs(case, seed)
    if kind == "uneven":
        cols = [[], [], []]
        for i, (nx, ny, nz, re, dt) in enumerate(_instances(case)):
            ch = _Channel(nx, ny, nz, case["lx"], case["lz"], re, dt)
            c, ics, ac = _exact_sweep(ch, inp["C"][i][0], list(inp["IC"][i]), inp["AC"][i][0], n, _inhomo(case),
                                      case["strength"])
            for col, parts in zip(cols, ([c], ics, [ac])):
                col += [p.reshape(-1) for p in parts]
        return [torch.cat(c).cpu().numpy() for c in cols]
    ch = _Channel(case["nx"], case["ny"], case["nz"], case["lx"], case["lz"], case["re"], case["dt"])
    if kind == "spec2phys":
        return [ch.velocity_values(inp["C"][0]).permute(0, 3, 2, 1).contiguous().cpu().numpy()]
    if kind == "gradient":
        c = inp["C"][0].clone().requires_grad_(True)
        nu = torch.tensor(1.0 / case["re"], dtype=torch.float64, device=c.device, requires_grad=True)
        flux = torch.tensor(FLUX, dtype=torch.float64, device=c.device, requires_grad=True)
        ch.nu = nu
        traj = ch.primal(c, n, cached=False, flux=flux)
        J = (torch.conj(inp["AC"][0]) * traj[-1]).real.sum()
        for i in range(n):
            J = J + (torch.conj(inp["src"][0]) * traj[3 * i]).real.sum()
        gc, gnu, gf = torch.autograd.grad(J, (c, nu, flux))
        # the mean-flux forcing is the derivative in the mean velocity (flux = 2 meanU), nu = 1 / Re
        return [traj[-1].detach().cpu().numpy(), gc.cpu().numpy(), 2 * float(gf), -float(gnu) / case["re"] ** 2]
    if kind == "kkt":
        return _exact_kkt(ch, inp["x"], case["segs"], n, _window_seed(case))
    nt, forced = case["ntan"], _inhomo(case) if case["ntan"] else []
    out = [[], [], []]
    for s in range(case["segs"]):
        ics = [inp["IC"][s * nt + j] for j in range(nt)]
        c, ends, ac = _exact_sweep(ch, inp["C"][s], ics, inp["AC"][s], n, forced, case["strength"])
        for col, parts in zip(out, ([c], ends, [ac])):
            col += parts
    if kind == "segments":
        return [_real(torch.stack(x)) for x in out]
    return [x.cpu().numpy() for col in out for x in col]
