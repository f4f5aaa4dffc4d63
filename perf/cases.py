"""The work a user of the library has it do, as timed cases.

A case is one pass of the RK4 step loop through a public entry point:

* ``solver`` -- a frame of a resident run: the state is loaded from device
  arrays, a chunk of steps is run, the new state is copied to device arrays
  (:class:`nlsemagic_gb300.api.Solver`);
* ``call`` -- the drop-in step function on host arrays, state in, state out
  (``NLSE{1,2,3}D_TAKE_STEPS_{CD,2SHOC}_CUDA_{F,D,M}``);
* ``batch`` -- a group of requests served together: admitted, advanced,
  fetched and released (:class:`nlsemagic_gb300.api.Batch`).

Classes: ``fp32``, ``fp64`` (the reference's bits), ``fma`` (FP64 with
contraction, what the serving loop runs its FP64 requests in) and ``mixed``.
Sizes are those of the benchmark, of the uneven batch and the serving stream,
and odd ones between; the data are the benchmark's: grey solitons in 1D,
vortices in 2D, vortex rings in a trap in 3D, with noise.
"""
import math
import random

import numpy as np
import torch

from nlsemagic_gb300 import _lib, api

SPACING = {1: 0.1, 2: 0.25, 3: 0.3}
PRECISION = {"fp32": 1, "fp64": 2, "fma": 2, "mixed": 3}
LETTER = {"fp32": "F", "fp64": "D", "mixed": "M"}
FLAG_FMA = 4


def _case(name, entry, shape, method, precision, bc, steps):
    shape = tuple(shape) + (1,) * (3 - len(shape))
    return {"name": name, "entry": entry, "ndim": sum(d > 1 for d in shape), "M": shape[0],
            "N": shape[1], "L": shape[2], "method": method, "precision": precision, "bc": bc,
            "steps": steps}


def _batch(name, count, mix, precision, steps):
    return {"name": name, "entry": "batch", "count": count, "mix": mix, "precision": precision,
            "steps": steps}


def listed():
    return [
        # the smallest drop-in call: one frame of the 1D research driver
        _case("call_1d_cd_fp64_1000", "call", (1000,), 1, "fp64", 2, 50),
        # the benchmark's 1D configuration (grey soliton, 1024 points, chunks of 100)
        _case("1d_cd_mixed_1024", "solver", (1024,), 1, "mixed", 2, 100),
        # a 1D request near the top of the serving range, a ragged size
        _case("1d_2shoc_mixed_48611", "solver", (48611,), 2, "mixed", 2, 100),
        # a long 1D domain in the reference's single precision
        _case("1d_cd_fp32_1000003", "solver", (1000003,), 1, "fp32", 3, 20),
        # the benchmark's 2D configuration (dark vortices, Dirichlet)
        _case("2d_2shoc_mixed_512", "solver", (512, 512), 2, "mixed", 1, 100),
        # a large 2D domain in single precision, odd sides
        _case("2d_cd_fp32_1537x1203", "solver", (1537, 1203), 1, "fp32", 2, 40),
        # the drop-in call on a small 2D grid in double precision
        _case("call_2d_2shoc_fp64_200x333", "call", (200, 333), 2, "fp64", 1, 50),
        # a 2D double-precision request as the serving loop runs it
        _case("2d_2shoc_fma_701x640", "solver", (701, 640), 2, "fma", 2, 20),
        # the headline configuration (vortex rings, 320^3, MSD)
        _case("3d_2shoc_mixed_320", "solver", (320, 320, 320), 2, "mixed", 2, 50),
        # a small 3D request, odd sides (rows that are no multiple of 16 bytes)
        _case("3d_2shoc_mixed_61x72x67", "solver", (61, 72, 67), 2, "mixed", 2, 100),
        # a 3D double-precision request as the serving loop runs it
        _case("3d_2shoc_fma_128", "solver", (128, 128, 128), 2, "fma", 1, 20),
        # uneven 1D and 2D requests served together
        _batch("batch_mixed_24", 24, 1003, "mixed", 300),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# point-steps a drawn case may take, by class: within the largest listed case's time
MOST = {"fp32": 7e8, "mixed": 7e8, "fma": 6e7, "fp64": 5e7}


def draw(rng):
    entry = rng.choice(["solver"] * 7 + ["call"] * 2 + ["batch"])
    if entry == "batch":
        c = _batch("", rng.randint(4, 32), rng.randint(0, 10 ** 6),
                   rng.choice(["mixed", "mixed", "fma"]), 0)
        c["steps"] = _log_int(rng, 50, 300)
        points = sum(_points(s) for s, _ in _batch_solves(c))
        c["steps"] = max(10, min(c["steps"], int(MOST[c["precision"]] / points)))
    else:
        precision = rng.choice(["fp32", "fp64", "mixed", "mixed"] +
                               (["fma"] if entry == "solver" else []))
        ndim = rng.choice([1, 1, 2, 2, 3])
        method = rng.choice([1, 2])
        bc = rng.choice([1, 1, 1, 2, 2, 2, 3] + ([4] if ndim == 1 else []))
        if ndim == 1:
            shape = (_log_int(rng, 300, 1000000),)
        elif ndim == 2:
            side = _log_int(rng, 64, 1300)
            shape = tuple(max(48, int(side * rng.uniform(0.8, 1.2))) for _ in range(2))
        else:
            side = _log_int(rng, 32, 250)
            shape = tuple(max(24, int(side * rng.uniform(0.8, 1.2))) for _ in range(3))
        if entry == "call" and _points(shape) > 500000:  # host copies count for both
            shape = tuple(max(24, int(d * (500000 / _points(shape)) ** (1 / ndim)))
                          for d in shape)
        steps = max(4, min(_log_int(rng, 20, 100), int(MOST[precision] / _points(shape))))
        c = _case("", entry, shape, method, precision, bc, steps)
    del c["name"]
    return c


def _points(shape):
    return math.prod(shape)


def _shape(case):
    return (case["M"], case["N"], case["L"])[:case["ndim"]]


def _time_step(ndim, method, a=1.0):
    """0.8 of the linear stability limit."""
    h = SPACING[ndim]
    return 0.8 * h * h / (ndim * math.sqrt(2.0) * a) * (0.75 if method == 2 else 1.0)


def _batch_solves(case):
    """(shape, method) of each request: 60% 1D, 40% square 2D, sizes log-uniform."""
    rng = random.Random(case["mix"])
    out = []
    for _ in range(case["count"]):
        if rng.random() < 0.6:
            shape = (_log_int(rng, 256, 16384),)
        else:
            shape = (_log_int(rng, 64, 512),) * 2
        out.append((shape, rng.choice([1, 2])))
    return out


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _field(shape, seed):
    """Initial state and potential on the device, slowest axis first (so that
    flattening gives the column-major order of the interface)."""
    ndim, h, dev = len(shape), SPACING[len(shape)], _device()
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=dev).manual_seed(int(rng.integers(1 << 31)))
    sides = tuple(reversed(shape))
    ax = []
    for d, n in enumerate(sides):
        x = (torch.arange(n, dtype=torch.float64, device=dev) - n / 2) * h
        ax.append(x.reshape([-1 if t == d else 1 for t in range(ndim)]))

    def noise(amount):
        return amount * torch.randn(sides, generator=gen, dtype=torch.float64, device=dev)

    if ndim == 1:  # grey soliton, the domain's middle half
        c = 0.5
        w = math.sqrt(1 - c * c / 2)
        x0 = float(rng.uniform(-0.25, 0.25)) * shape[0] * h
        U = torch.complex(w * torch.tanh(w * (ax[0] - x0) / math.sqrt(2)) + noise(1e-4),
                          c / math.sqrt(2) + noise(1e-4))
        return U, torch.zeros(sides, dtype=torch.float64, device=dev)
    if ndim == 2:  # four vortices of charge +-1, phase noise
        U = torch.ones(sides, dtype=torch.complex128, device=dev)
        for t in range(4):
            dy = ax[0] - float(rng.uniform(-0.16, 0.16)) * sides[0] * h
            dx = ax[1] - float(rng.uniform(-0.16, 0.16)) * sides[1] * h
            U = U * torch.polar(torch.tanh(torch.hypot(dx, dy)),
                                (1 - 2 * (t % 2)) * torch.atan2(dy, dx))
        return (U * torch.polar(torch.ones_like(U.real), noise(1e-3)),
                torch.zeros(sides, dtype=torch.float64, device=dev))
    # four vortex rings on a Thomas-Fermi background in a harmonic trap
    size = max(sides) * h
    omega = 0.02 * 96.0 / size
    V = 0.5 * omega * omega * (ax[0] ** 2 + ax[1] ** 2 + ax[2] ** 2)
    U = torch.sqrt(torch.clamp(1.0 - V, min=0.0)).to(torch.complex128)
    for _ in range(4):
        radius = float(rng.uniform(0.06, 0.1)) * size
        at = rng.uniform(-0.16, 0.16, size=3) * size
        n = rng.standard_normal(3)
        n /= np.linalg.norm(n)
        dz, dy, dx = (ax[d] - float(at[d]) for d in range(3))
        along = dz * float(n[0]) + dy * float(n[1]) + dx * float(n[2])
        dr = torch.sqrt(torch.clamp(dz * dz + dy * dy + dx * dx - along * along, min=0.0)) - radius
        U = U * torch.polar(torch.tanh(torch.hypot(dr, along)), torch.atan2(along, dr))
    return U, V.contiguous()


def _host(T):
    """A device field as the MATLAB-shaped host array."""
    return np.asfortranarray(T.cpu().numpy().transpose())


def _flags(precision):
    return _lib.FLAG_MSD_GUARD | (FLAG_FMA if precision == "fma" else 0)


def prepare(case, seed):
    if case["entry"] == "batch":
        solves = []
        for t, (shape, method) in enumerate(_batch_solves(case)):
            U, V = _field(shape, seed * 1000 + t)
            solves.append((_host(U), _host(V), method))
        need = sum(api.Batch.bytes_for(U.shape, PRECISION[case["precision"]]) for U, _, _ in solves)
        pool = api.Batch(need + (1 << 20) * len(solves), max_solves=len(solves))
        return {"case": case, "pool": pool, "solves": solves}
    shape = _shape(case)
    U, V = _field(shape, seed)
    if case["entry"] == "call":
        f = getattr(api, "NLSE%dD_TAKE_STEPS_%s_CUDA_%s" % (
            case["ndim"], "CD" if case["method"] == 1 else "2SHOC", LETTER[case["precision"]]))
        return {"case": case, "call": f, "U": _host(U), "V": _host(V)}
    h = SPACING[case["ndim"]]
    solver = api.Solver(shape, method=case["method"], precision=PRECISION[case["precision"]],
                        BC=case["bc"], s=-1.0, a=1.0, h2=h * h,
                        k=_time_step(case["ndim"], case["method"]),
                        flags=_flags(case["precision"]))
    re, im = U.real.contiguous(), U.imag.contiguous()
    return {"case": case, "solver": solver, "re": re, "im": im, "V": V,
            "out": (torch.empty_like(re), torch.empty_like(im))}


def run(state):
    case = state["case"]
    if case["entry"] == "solver":
        s, out = state["solver"], state["out"]
        s.upload_device(state["re"].data_ptr(), state["im"].data_ptr(), state["V"].data_ptr())
        s.run(case["steps"])
        s.download_device(out[0].data_ptr(), out[1].data_ptr())
        return out
    if case["entry"] == "call":
        h = SPACING[case["ndim"]]
        return state["call"](state["U"], state["V"], -1.0, 1.0, h * h, case["bc"], case["steps"],
                             _time_step(case["ndim"], case["method"]))
    pool = state["pool"]
    slots = []
    for U, V, method in state["solves"]:
        h = SPACING[U.ndim]
        slots.append(pool.add(U, V, -1.0, 1.0, h * h, 2, case["steps"],
                              _time_step(U.ndim, method), method=method,
                              precision=PRECISION[case["precision"]],
                              flags=_flags(case["precision"])))
    pool.run(case["steps"])
    out = [pool.download(t) for t in slots]
    for t in slots:
        pool.remove(t)
    return out


def work(case):
    """State and potential read once (planar doubles), the new state written
    once; per point and stage the operations of the stencil (neighbour sums,
    weights), the local term and the RK4 update."""
    if case["entry"] == "batch":
        solves = _batch_solves(case)
    else:
        solves = [(_shape(case), case["method"])]
    b = f = 0
    for shape, method in solves:
        d, n = len(shape), _points(shape)
        stencil = 2 * (2 * d + 2) if method == 1 else 2 * (4 * d + 3)
        b += n * (24 + 16)
        f += n * case["steps"] * 4 * (stencil + 5 + 4 + 6)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same steps in plain 64-bit torch
# ---------------------------------------------------------------------------
def _shift(U, by):
    """U moved by `by` (one offset per axis), the interior part."""
    return U[tuple(slice(1 + d, U.shape[t] - 1 + d) for t, d in enumerate(by))]


def _unit(ndim):
    for t in range(ndim):
        for d in (1, -1):
            yield tuple(d if t == u else 0 for u in range(ndim))


def _diagonal(ndim):
    """Neighbours one cell off along two axes each."""
    for t in range(ndim):
        for u in range(t):
            for d in (1, -1):
                for e in (1, -1):
                    yield tuple(d if x == t else e if x == u else 0 for x in range(ndim))


def _ends(U, h2):
    """One-sided second differences at the two ends (1D)."""
    return ((2 * U[0] - 5 * U[1] + 4 * U[2] - U[3]) / h2,
            (2 * U[-1] - 5 * U[-2] + 4 * U[-3] - U[-4]) / h2)


class _Rhs:
    def __init__(self, V, bc, method, h2, s=-1.0, a=1.0):
        self.V, self.bc, self.method, self.h2, self.s, self.a = V, bc, method, h2, s, a
        d = V.ndim
        self.inner = (slice(1, -1),) * d
        self.clamp = [torch.arange(n, device=V.device).clamp(1, n - 2) for n in V.shape]
        self.zero = (0,) * d

    def neighbour(self, X):
        """X at each point's interior neighbour (itself, if interior)."""
        for t, i in enumerate(self.clamp):
            X = X.index_select(t, i)
        return X

    def faces(self):
        """The boundary as slices of the grid."""
        for t in range(self.V.ndim):
            for e in (slice(0, 1), slice(-1, None)):
                yield tuple(e if x == t else slice(None) for x in range(self.V.ndim))

    def at_faces(self, full, value):
        """Sets full[f] = value(f, clamped picker) on every face f."""
        for t, f in enumerate(self.faces()):
            def q(X, f=f, axis=t // 2, side=t % 2):
                n = X.shape[axis]
                Y = X.narrow(axis, n - 2 if side else 1, 1)
                for u, i in enumerate(self.clamp):
                    if u != axis:
                        Y = Y.index_select(u, i)
                return Y
            full[f] = value(f, q)
        return full

    def ratio(self, num, Uq):
        den = Uq.real ** 2 + Uq.imag ** 2
        zero = (Uq.real == 0) & (Uq.imag == 0)
        return torch.where(zero, torch.zeros_like(den), num / torch.where(zero, 1.0, den))

    def __call__(self, U):
        d, a, h2, V, bc = self.V.ndim, self.a, self.h2, self.V, self.bc
        N = self.s * (U.real ** 2 + U.imag ** 2) - V
        U0 = U[self.inner]
        D0 = sum(_shift(U, o) - U0 for o in _unit(d)) / h2
        if self.method == 1:
            lap = D0
        else:
            D = torch.zeros_like(U)
            D[self.inner] = D0
            if bc == 4:
                D[0], D[-1] = _ends(U, h2)
            elif bc == 1:
                self.at_faces(D, lambda f, q: -N[f] / a * U[f])
            elif bc == 2:
                Dint = D.clone()

                def msd(f, q):
                    Uq, Dq = q(U), q(Dint)
                    A = self.ratio(Dq.real * Uq.real + Dq.imag * Uq.imag, Uq)
                    return (A + (q(N) - N[f]) / a) * U[f]
                self.at_faces(D, msd)
            near = sum(_shift(D, o) for o in _unit(d))
            if d == 1:
                lap = (14 * D0 - near) / 12
            else:
                diag = sum(_shift(U, o) - U0 for o in _diagonal(d)) / h2
                lap = ((12 if d == 2 else 10) * D0 - near + 2 * diag) / 12
        F = torch.zeros_like(U)
        F[self.inner] = 1j * (a * lap + N[self.inner] * U0)
        if bc == 2:
            Fint = F.clone()

            def msd(f, q):
                Uq, Fq = q(U), q(Fint)
                return 1j * self.ratio(Fq.imag * Uq.real - Fq.real * Uq.imag, Uq) * U[f]
            self.at_faces(F, msd)
        elif bc == 3:
            self.at_faces(F, lambda f, q: 1j * N[f] * U[f])
        elif bc == 4:
            e0, e1 = _ends(U, h2)
            F[0], F[-1] = 1j * (a * e0 + N[0] * U[0]), 1j * (a * e1 + N[-1] * U[-1])
        return F


def _steps(U, V, bc, method, steps):
    h = SPACING[V.ndim]
    k = _time_step(V.ndim, method)
    rhs = _Rhs(V, bc, method, h * h)
    for _ in range(steps):
        F = rhs(U)
        S = F
        F = rhs(U + 0.5 * k * F)
        S = S + 2 * F
        F = rhs(U + 0.5 * k * F)
        S = S + 2 * F
        F = rhs(U + k * F)
        U = U + k / 6 * (S + F)
    return U


def exact(case, seed):
    if case["entry"] == "batch":
        out = []
        for t, (shape, method) in enumerate(_batch_solves(case)):
            U, V = _field(shape, seed * 1000 + t)
            out.append(_host(_steps(U, V, 2, method, case["steps"])))
        return out
    U, V = _field(_shape(case), seed)
    U = _steps(U, V, case["bc"], case["method"], case["steps"])
    if case["entry"] == "call":
        return _host(U)
    return U.real.contiguous(), U.imag.contiguous()
