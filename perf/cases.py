"""Performance cases of the channel time step: what a user of this package has it do.

Every case goes through the package's public entry points (``Channel``,
``Ensemble``, ``Mlp``) on a field that lies in host memory at the start, as a
restart file does.  ``step`` cases take whole RK3 steps with their Runtimedata
line each, as the driver's time loop does, then fetch the field into a pinned
buffer, as a run does that writes its fields; ``ensemble`` cases advance many
small channels together; ``closure`` cases step a coarse channel with the
learned subgrid stresses; ``budget`` cases add one sample to the
Reynolds-stress budget spectra and read them.

``exact`` restates the same work with torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

RK = ((120.0 / 32.0, 2.0, 0.0), (120.0 / 8.0, 50.0 / 8.0, 34.0 / 8.0), (120.0 / 20.0, 90.0 / 20.0, 50.0 / 20.0))
PRECISIONS = ("fp64", "fp64dd", "mixed")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest run that the repository configures: fixed time step, launches and latency count
        {"name": "small fp64", "kind": "step", "nx": 32, "ny": 64, "nz": 32, "alfa0": 1.0, "beta0": 2.0, "re": 4000.0,
         "a": 1.6, "deltat": 0.004, "cflmax": 0.0, "precision": "fp64", "steps": 2},
        # the coarse grid of the subgrid closure, without it: few (kx, kz) pairs for the solves
        {"name": "coarse mixed", "kind": "step", "nx": 47, "ny": 96, "nz": 47, "alfa0": 1.0, "beta0": 2.0, "re": 4200.0,
         "a": 1.6, "deltat": 0.0, "cflmax": 1.0, "precision": "mixed", "steps": 2},
        # sizes off the tuned ones: padded lengths 128 and 256, odd row counts
        {"name": "uneven fp64", "kind": "step", "nx": 79, "ny": 101, "nz": 75, "alfa0": 0.7, "beta0": 1.5, "re": 3000.0,
         "a": 1.5, "deltat": 0.0, "cflmax": 1.0, "precision": "fp64", "steps": 2},
        {"name": "uneven mixed", "kind": "step", "nx": 83, "ny": 120, "nz": 85, "alfa0": 0.6, "beta0": 1.3, "re": 5000.0,
         "a": 1.7, "deltat": 0.0, "cflmax": 1.0, "precision": "mixed", "steps": 2},
        # the Re_tau = 180 channel in its three precisions
        {"name": "retau180 fp64", "kind": "step", "nx": 127, "ny": 192, "nz": 127, "alfa0": 0.5, "beta0": 1.0,
         "re": 4200.0, "a": 1.6, "deltat": 0.0, "cflmax": 1.0, "precision": "fp64", "steps": 2},
        {"name": "retau180 fp64dd", "kind": "step", "nx": 127, "ny": 192, "nz": 127, "alfa0": 0.5, "beta0": 1.0,
         "re": 4200.0, "a": 1.6, "deltat": 0.0, "cflmax": 1.0, "precision": "fp64dd", "steps": 2},
        {"name": "retau180 mixed", "kind": "step", "nx": 127, "ny": 192, "nz": 127, "alfa0": 0.5, "beta0": 1.0,
         "re": 4200.0, "a": 1.6, "deltat": 0.0, "cflmax": 1.0, "precision": "mixed", "steps": 2},
        # a large channel in full precision
        {"name": "large fp64", "kind": "step", "nx": 255, "ny": 256, "nz": 255, "alfa0": 0.5, "beta0": 1.0,
         "re": 10000.0, "a": 1.8, "deltat": 0.0, "cflmax": 1.0, "precision": "fp64", "steps": 1},
        # the Re_tau = 550 channel of the benchmark, mixed precision
        {"name": "retau550 mixed", "kind": "step", "nx": 383, "ny": 384, "nz": 383, "alfa0": 0.5, "beta0": 1.0,
         "re": 14000.0, "a": 1.8, "deltat": 0.0, "cflmax": 1.0, "precision": "mixed", "steps": 1},
        # the batched ensemble: 64 uneven minimal channels, one launch for a step of all
        {"name": "ensemble mixed", "kind": "ensemble", "members": 64, "precision": "mixed", "steps": 4},
        # the coarse run with the network in every convolution pass
        {"name": "closure fp64", "kind": "closure", "nx": 47, "ny": 96, "nz": 47, "alfa0": 1.0, "beta0": 2.0,
         "re": 4200.0, "a": 1.6, "deltat": 0.005, "cflmax": 0.0, "precision": "fp64", "steps": 1},
        # post-processing during the run: one sample of the budget spectra, then the spectra
        {"name": "budget fp64", "kind": "budget", "nx": 127, "ny": 192, "nz": 127, "alfa0": 0.5, "beta0": 1.0,
         "re": 4200.0, "a": 1.6, "deltat": 0.0, "cflmax": 1.0, "precision": "fp64", "steps": 0},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("step", "ensemble", "closure", "budget"), (9, 1, 1, 1))[0]
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(5, 48), "precision": rng.choice(PRECISIONS), "steps": rng.randint(1, 4)}
    small = kind != "step"
    nx, nz = _logint(rng, 16, 64 if small else 255), _logint(rng, 16, 64 if small else 255)
    ny = _logint(rng, 40, 128 if small else 256)
    alfa0, beta0 = round(rng.uniform(0.4, 2.0), 3), round(rng.uniform(0.8, 4.0), 3)
    # a Reynolds number that the grid resolves about as well as the listed channels do
    re = rng.uniform(30.0, 70.0) * min(nx * alfa0, nz * beta0, 0.7 * ny)
    fixed = kind == "closure" or rng.random() < 0.2
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "alfa0": alfa0, "beta0": beta0, "re": round(re, 1),
            "a": round(rng.uniform(1.4, 1.9), 3), "deltat": 0.001 if fixed else 0.0, "cflmax": 0.0 if fixed else 1.0,
            "precision": rng.choice(PRECISIONS), "steps": 0 if kind == "budget" else rng.randint(1, 2)}


# ---------------------------------------------------------------------------
# inputs, the same in numpy for the run and for its restatement
# ---------------------------------------------------------------------------
def _members(case, seed):
    """The uneven minimal channels of an ensemble case, as step cases."""
    size = np.random.default_rng(case["members"])
    r = np.random.default_rng([seed, case["members"]])
    out = []
    for _ in range(case["members"]):
        nx, nz = (int(v) for v in size.choice([16, 24, 32], size=2))
        out.append({"kind": "step", "nx": nx, "ny": int(size.choice([48, 64, 96])), "nz": nz,
                    "alfa0": float(r.uniform(1.0, 2.0)), "beta0": float(r.uniform(2.0, 4.0)),
                    "re": float(r.uniform(2000.0, 4000.0)), "a": 1.6, "deltat": 0.004, "cflmax": 0.0,
                    "precision": case["precision"], "steps": case["steps"]})
    return out


def _y(c):
    iy = np.arange(-1, c["ny"] + 2, dtype=np.float64)
    return np.tanh(c["a"] * (2.0 * iy / c["ny"] - 1.0)) / math.tanh(c["a"]) + 1.0


def _modes(c, seed, cut=32, amplitude=0.03):
    """A laminar profile with a divergence-free perturbation of every mode up
    to |kx|, |kz| = cut whose amplitude falls with the wavenumber:
    (3, K+1, 2L+1, ny+3) complex, the modes kx = 0..K, kz = -L..L."""
    K, L = min(cut, c["nx"]), min(cut, c["nz"])
    r = np.random.default_rng([seed, c["nx"], c["ny"], c["nz"]])
    s = _y(c)
    base = s * (2.0 - s)
    dbase = 4.0 * base * (1.0 - s)  # d/dy of base^2
    jx, jz = np.arange(K + 1)[:, None], np.arange(-L, L + 1)[None, :]
    kx, kz = c["alfa0"] * jx, c["beta0"] * jz
    k2 = kx * kx + kz * kz
    k2[0, L] = 1.0
    amp = amplitude * (1.0 + (jx * jx + jz * jz) / 4.0) ** -1.25
    ph = np.exp(2j * np.pi * r.random((2, K + 1, 2 * L + 1)))
    cv, ce = (amp * ph[0])[..., None], (amp * ph[1])[..., None]
    v, dv, eta = cv * base**2, cv * dbase, ce * base
    ax, az, q = 1j * kx[..., None], 1j * kz[..., None], k2[..., None]
    V = np.stack([(ax * dv - az * eta) / q, v, (az * dv + ax * eta) / q])
    V[:, 0, :L] = np.conj(V[:, 0, :L:-1])  # a real field
    V[:, 0, L] = 0.0
    V[0, 0, L] = base
    return V


def _field(c, seed):
    V = np.zeros((3, c["nx"] + 1, 2 * c["nz"] + 1, c["ny"] + 3), dtype=np.complex128)
    m = _modes(c, seed)
    K, L = m.shape[1] - 1, m.shape[2] // 2
    V[:, : K + 1, c["nz"] - L : c["nz"] + L + 1] = m
    return V


def _network(seed):
    """Weights (the parameter vector of include/chgpu_closure.h) and scales of a small trained-like network."""
    r = np.random.default_rng([seed, 77])
    W1 = r.standard_normal((64, 16)) * 0.3
    W1[:, 11:] = 0.0
    parts = [W1, r.standard_normal((64, 64)) / 8.0, r.standard_normal(64) * 0.1, r.standard_normal((64, 64)) / 8.0,
             r.standard_normal(64) * 0.1, r.standard_normal((6, 64)) / 8.0, r.standard_normal(6) * 0.1]
    theta = np.concatenate([p.ravel() for p in parts]).astype(np.float32)
    f = np.float32
    norm = {"mu_in": np.zeros(10, f), "sd_in": np.array([1, 2, 1, 1, 1, 1, 1, 1, 1, 0.5], f),
            "mu_out": np.zeros(6, f), "sd_out": np.full(6, 1e-4, f)}
    return theta, norm


def _dns(c):
    from channel_gb300 import DnsIn

    return DnsIn(nx=c["nx"], ny=c["ny"], nz=c["nz"], alfa0=c["alfa0"], beta0=c["beta0"], re=c["re"], a=c["a"],
                 ymin=0.0, ymax=2.0, meanflowx=4.0 / 3.0, deltat=c["deltat"], cflmax=c["cflmax"], nstep=c["steps"])


def _pinned(n):
    return torch.empty(n, dtype=torch.complex128, pin_memory=True).numpy()


def prepare(case, seed):
    from channel_gb300 import Channel, Ensemble

    if case["kind"] == "ensemble":
        members = _members(case, seed)
        ens = Ensemble([_dns(c) for c in members], case["precision"])
        for i, (c, m) in enumerate(zip(members, ens.members)):
            m.upload(_field(c, seed + i))
            m.start()
        sizes = [int(np.prod(m.shape)) for m in ens.members]
        out = _pinned(sum(sizes))
        at = np.cumsum([0] + sizes)
        views = [out[at[i]:at[i + 1]].reshape(m.shape) for i, m in enumerate(ens.members)]
        return {"kind": "ensemble", "ens": ens, "out": out, "views": views, "steps": case["steps"]}
    g = Channel(_dns(case), case["precision"])
    V = _field(case, seed)
    g.upload(V)
    g.start()
    state = {"kind": case["kind"], "g": g, "steps": case["steps"]}
    if case["kind"] == "budget":
        g.tke_reset(V[0, 0, case["nz"]].real.copy(), np.zeros(case["ny"] + 3))
        state["mean"] = V[0, 0, case["nz"]].real.copy()
        return state
    if case["kind"] == "closure":
        from channel_gb300 import closure

        net = closure.Mlp(0)
        net.params, net.norm = _network(seed)
        g.closure_attach(net)
        state["net"] = net
    state["out"] = _pinned(int(np.prod(g.shape))).reshape(g.shape)
    return state


def run(state):
    if state["kind"] == "ensemble":
        ens = state["ens"]
        for _ in range(state["steps"]):
            lines = ens.step()
        for m, v in zip(ens.members, state["views"]):
            m.download(v)
        return [state["out"], np.stack(lines)]
    g = state["g"]
    if state["kind"] == "budget":
        g.tke_reset(state["mean"], np.zeros(state["mean"].size))
        g.tke_accumulate()
        mean, spectra, profiles, _ = g.tke_result()
        return [mean, spectra, profiles]
    lines = [g.step() for _ in range(state["steps"])]
    return [g.download(state["out"]), np.stack(lines)]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _fit(n):
    while True:
        j = n
        while j % 2 == 0:
            j >>= 1
        if j in (1, 3):
            return n
        n += 1


def _padded(c):
    return _fit(3 * (c["nx"] + 1) // 2), _fit(3 * c["nz"])


def _transforms(c, fields):
    """Operations of the padded transforms of that many fields over all planes (5/2 n log2 n for n real points)."""
    nxd, nzd = _padded(c)
    z = (c["nx"] + 1) * 5.0 * nzd * math.log2(nzd)
    x = nzd * 2.5 * 2 * nxd * math.log2(2 * nxd)
    return fields * (z + x) * (c["ny"] + 3)


def _step_work(c):
    """One RK3 step: each substep reads and writes the field (three complex
    numbers a point, 64 bits) and the explicit terms it keeps (two, in the
    precision's own type); nine transforms, six products, about 500
    operations a point for the wall-normal stencils, the two banded
    factorisations and solves and the velocity recovery."""
    points = (c["nx"] + 1) * (2 * c["nz"] + 1) * (c["ny"] + 3)
    nxd, nzd = _padded(c)
    kept = 8 if c["precision"] == "mixed" else 16
    products = 6.0 * 2 * nxd * nzd * (c["ny"] + 3)
    return 3.0 * points * (2 * 48 + 4 * kept), 3.0 * (_transforms(c, 9) + products + 500.0 * points)


def work(case):
    if case["kind"] == "ensemble":
        each = [_step_work(c) for c in _members(case, 0)]
        return {"bytes": case["steps"] * sum(e[0] for e in each), "flops": case["steps"] * sum(e[1] for e in each)}
    points = (case["nx"] + 1) * (2 * case["nz"] + 1) * (case["ny"] + 3)
    if case["kind"] == "budget":
        out = 8.0 * 60 * (2 * case["nz"] + 1) * (case["ny"] + 3)
        return {"bytes": 48.0 * points + out, "flops": _transforms(case, 15) + 300.0 * points}
    b, f = _step_work(case)
    if case["kind"] == "closure":  # nine gradients to the points, 9.5 k multiply-adds of the network a point
        nxd, nzd = _padded(case)
        f += 3.0 * (_transforms(case, 9) + 2.0 * 9500 * 2 * nxd * nzd * (case["ny"] - 1))
    return {"bytes": case["steps"] * b, "flops": case["steps"] * f}


# ---------------------------------------------------------------------------
# the same in 64 bits with torch
# ---------------------------------------------------------------------------
def _weights(dy, powers):
    """w with sum_j w_j dy_j^i = powers[i], i = 0..4, solved in extended precision."""
    dy = np.asarray(dy, np.longdouble)
    h = np.abs(dy).max()
    A = np.array([(dy / h) ** i for i in range(5)], np.longdouble)
    b = np.array([np.longdouble(p) / h**i for i, p in enumerate(powers)], np.longdouble)
    for i in range(5):  # Gaussian elimination with pivoting
        k = i + int(np.argmax(np.abs(A[i:, i])))
        A[[i, k]], b[[i, k]] = A[[k, i]], b[[k, i]]
        for r in range(i + 1, 5):
            f = A[r, i] / A[i, i]
            A[r] -= f * A[i]
            b[r] -= f * b[i]
    x = np.zeros(5, np.longdouble)
    for i in range(4, -1, -1):
        x[i] = (b[i] - (A[i, i + 1:] * x[i + 1:]).sum()) / A[i, i]
    return x


class _Stencils:
    """Compact five-point stencils on the stretched grid: with d4 the fourth
    derivative of the quartic through five points, d0 such that d0 f = d4 of
    the fourth integral of f, and d1, d2 the stencils with d0 f' = d1 f and
    d0 f'' = d2 f for quartic f; one-sided first and second derivatives at the
    walls and ghost points."""

    def __init__(self, c):
        ny = self.ny = c["ny"]
        y = self.y = _y(c).astype(np.longdouble)
        d = np.zeros((ny + 1, 4, 5), np.longdouble)  # rows iy: d0, d1, d2, d4
        for iy in range(1, ny):
            dy = y[iy - 1:iy + 4] - y[iy + 1]
            d4 = _weights(dy, [0, 0, 0, 0, 24])
            # d0 of dy^i is d4 of dy^(i+4) over (i+1)(i+2)(i+3)(i+4)
            d0 = _weights(dy, [(d4 * dy ** (i + 4)).sum() / ((i + 1) * (i + 2) * (i + 3) * (i + 4)) for i in range(5)])
            d1 = _weights(dy, [0] + [(d0 * i * dy ** (i - 1)).sum() for i in range(1, 5)])
            d2 = _weights(dy, [0, 0] + [(d0 * i * (i - 1) * dy ** (i - 2)).sum() for i in range(2, 5)])
            d[iy] = d0, d1, d2, d4
        self.d = d.astype(np.float64)
        lo, hi = y[0:5], y[ny - 2:ny + 3]  # iy = -1..3 and ny-3..ny+1
        one, two = [0, 1, 0, 0, 0], [0, 0, 2, 0, 0]
        f = lambda rows, at, p: _weights(rows - at, p).astype(np.float64)  # noqa: E731
        # first and second derivatives at iy = -1, 0, ny, ny+1
        self.w1 = [f(lo, y[0], one), f(lo, y[1], one), f(hi, y[ny + 1], one), f(hi, y[ny + 2], one)]
        self.w2 = [f(lo, y[0], two), f(lo, y[1], two), f(hi, y[ny + 1], two), f(hi, y[ny + 2], two)]
        yy = y.astype(np.float64)
        w = np.zeros(ny + 3)  # the integral over y: a parabola through each pair of intervals
        for iy in range(1, ny, 2):
            p, m = yy[iy + 2] - yy[iy + 1], yy[iy] - yy[iy + 1]
            a1 = -m / 3 + p / 6 + p * p / (6 * m)
            a3 = p / 3 - m / 6 - m * m / (6 * p)
            w[iy], w[iy + 2] = w[iy] + a1, w[iy + 2] + a3
            w[iy + 1] += p - m - a1 - a3
        self.wint = w
        self.dy = np.zeros(ny + 3)
        self.dy[2:ny + 1] = 0.5 * (yy[3:ny + 2] - yy[1:ny])

    def rows(self, k, F):
        """sum_j d_k[iy][j] F(iy - 2 + j) for iy = 1..ny-1; F has rows iy = -1..ny+1."""
        n = self.ny - 1
        w = torch.as_tensor(self.d[1:self.ny, k], device=F.device)
        sh = (n,) + (1,) * (F.dim() - 1)
        return sum(w[:, j].reshape(sh) * F[j:j + n] for j in range(5))

    def ends(self, w, F):
        t = [torch.as_tensor(x, device=F.device).reshape((5,) + (1,) * (F.dim() - 1)) for x in w]
        lo, hi = F[0:5], F[-5:]
        return [(t[0] * lo).sum(0), (t[1] * lo).sum(0), (t[2] * hi).sum(0), (t[3] * hi).sum(0)]

    def derivative(self, F, order=1):
        """The compact derivative on all rows -1..ny+1."""
        e = self.ends(self.w1 if order == 1 else self.w2, F)
        b = self.rows(order, F)
        d0 = self.d[:, 0]
        ny = self.ny
        b[0] -= d0[1, 0] * e[0] + d0[1, 1] * e[1]
        b[1] -= d0[2, 0] * e[1]
        b[-1] -= d0[ny - 1, 3] * e[2] + d0[ny - 1, 4] * e[3]
        b[-2] -= d0[ny - 2, 4] * e[2]
        A = torch.as_tensor(d0[1:ny], device=F.device)[:, :, None].clone()
        x = _banded(A, b.reshape(ny - 1, -1)).reshape(b.shape)
        return torch.cat([e[0][None], e[1][None], x, e[2][None], e[3][None]])


def _banded(A, b):
    """x of the pentadiagonal systems A (rows, 5, systems or 1), b (rows, systems)."""
    n = b.shape[0]
    zero = torch.zeros_like(A[0, 0])
    U1, U2, x = [], [], []
    l1 = l2 = None
    for i in range(n):
        a0, a1, a2, a3, a4 = A[i]
        r = b[i]
        if i > 1:  # eliminate x(i-2) = x[i-2] - U1 x(i-1) - U2 x(i)
            a1, a2 = a1 - a0 * U1[i - 2], a2 - a0 * U2[i - 2]
            r = r - a0 * l2
        if i > 0:
            a2, a3 = a2 - a1 * U1[i - 1], a3 - a1 * U2[i - 1]
            r = r - a1 * l1
        U1.append(a3 / a2 if i < n - 1 else zero)
        U2.append(a4 / a2 if i < n - 2 else zero)
        l2, l1 = l1, r / a2
        x.append(l1)
    for i in range(n - 2, -1, -1):
        x[i] = x[i] - U1[i] * x[i + 1] - (U2[i] * x[i + 2] if i < n - 2 else 0.0)
    return torch.stack(x)


class _Exact:
    """One channel, rows iy = -1..ny+1 first: V (3, ny+3, nx+1, 2nz+1)."""

    def __init__(self, c, seed):
        self.c, self.st = c, _Stencils(c)
        self.nxd, self.nzd = _padded(c)
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        nx, nz, ny = c["nx"], c["nz"], c["ny"]
        m = torch.as_tensor(_modes(c, seed), device=self.dev).permute(0, 3, 1, 2)
        K, L = m.shape[2] - 1, m.shape[3] // 2
        self.V = torch.zeros((3, ny + 3, nx + 1, 2 * nz + 1), dtype=torch.complex128, device=self.dev)
        self.V[:, :, : K + 1, nz - L:nz + L + 1] = m
        f64 = {"dtype": torch.float64, "device": self.dev}
        self.kx = c["alfa0"] * torch.arange(nx + 1, **f64)[:, None]
        self.kz = c["beta0"] * torch.arange(-nz, nz + 1, **f64)[None, :]
        self.k2 = self.kx**2 + self.kz**2
        self.ni = 1.0 / c["re"]
        self.old = [0.0, 0.0]
        self.px = 0.0  # the pressure gradient that keeps the flow rate
        self.time, self.net = 0.0, None

    def physical(self, F):
        """(planes, nx+1, 2nz+1) to (planes, nzd, 2 nxd)."""
        nz = self.c["nz"]
        Z = torch.zeros(F.shape[:2] + (self.nzd,), dtype=F.dtype, device=F.device)
        Z[..., : nz + 1], Z[..., self.nzd - nz:] = F[..., nz:], F[..., :nz]
        Z = torch.fft.ifft(Z, dim=2, norm="forward").transpose(1, 2)
        X = torch.zeros(Z.shape[:2] + (self.nxd + 1,), dtype=F.dtype, device=F.device)
        X[..., : F.shape[1]] = Z
        X[..., 0].imag.zero_()
        return torch.fft.irfft(X, n=2 * self.nxd, dim=2, norm="forward")

    def spectral(self, R):
        nz = self.c["nz"]
        X = torch.fft.rfft(R, dim=2, norm="forward")[..., : self.c["nx"] + 1].transpose(1, 2)
        Z = torch.fft.fft(X, dim=2, norm="forward")
        return torch.cat([Z[..., self.nzd - nz:], Z[..., : nz + 1]], dim=2)

    def chunks(self):
        n = max(1, int(4e8 / (self.nzd * 2 * self.nxd * 8)))
        return [slice(i, min(i + n, self.c["ny"] + 3)) for i in range(0, self.c["ny"] + 3, n)]

    def gradient(self):
        G = []
        for F in self.V:
            G += [1j * self.kx * F, self.st.derivative(F), 1j * self.kz * F]
        return G

    def convolve(self, products=True):
        """The six products' spectra and the largest CFL number."""
        ny = self.c["ny"]
        rdx, rdz = self.c["alfa0"] * self.nxd / math.pi, self.c["beta0"] * self.nzd / (2 * math.pi)
        dy = torch.as_tensor(self.st.dy, device=self.dev)
        out, cfl = [[] for _ in range(6)], 0.0
        G = self.gradient() if self.net is not None and products else None
        for s in self.chunks():
            u, v, w = (self.physical(F[s]) for F in self.V)
            lo, hi = max(s.start, 2), min(s.stop, ny + 1)  # planes iy = 1..ny-1
            if lo < hi:
                q = slice(lo - s.start, hi - s.start)
                cfl = max(cfl, float((u[q].abs() * rdx + v[q].abs() / dy[lo:hi, None, None] + w[q].abs() * rdz).max()))
            if products:
                p = [u * u, v * v, w * w, u * v, v * w, u * w]
                if G is not None and lo < hi:
                    for a, t in zip(p, self.stresses([self.physical(g[lo:hi]) for g in G], lo, hi)):
                        a[q] += t
                for o, a in zip(out, p):
                    o.append(self.spectral(a))
        return [torch.cat(o) for o in out] if products else None, cfl

    def stresses(self, g, lo, hi):
        theta, norm = self.net
        t = torch.as_tensor(theta.astype(np.float64), device=self.dev)
        y = self.st.y.astype(np.float64)[lo:hi]
        wall = torch.as_tensor(np.minimum(y, 2.0 - y), device=self.dev)[:, None, None].expand(g[0].shape)
        n = {k: torch.as_tensor(v.astype(np.float64), device=self.dev) for k, v in norm.items()}
        W1, W2, b2, W3, b3, W4, b4 = torch.split(t, [1024, 4096, 64, 4096, 64, 384, 6])
        tau = torch.empty((6,) + g[0].shape, dtype=torch.float64, device=self.dev)
        act = torch.nn.functional.silu
        for i in range(hi - lo):
            x = torch.stack([f[i].reshape(-1) for f in g] + [wall[i].reshape(-1)])
            x = (x - n["mu_in"][:, None]) / n["sd_in"][:, None]
            x = torch.cat([x, torch.ones_like(x[:1])])
            h = act(W1.reshape(64, 16)[:, :11] @ x)
            h = act(W2.reshape(64, 64) @ h + b2[:, None])
            h = act(W3.reshape(64, 64) @ h + b3[:, None])
            o = (W4.reshape(6, 64) @ h + b4[:, None]) * n["sd_out"][:, None] + n["mu_out"][:, None]
            tau[:, i] = o.reshape(6, *g[0].shape[1:])
        return tau

    def solve(self, lam, b, which, wall=None):
        """v (which 0) or eta (1) on rows -1..ny+1 from the right-hand sides b (rows 1..ny-1)."""
        st, ny, ni = self.st, self.c["ny"], self.ni
        d = torch.as_tensor(st.d[1:ny], device=self.dev)[:, :, :, None]  # (rows, 4, 5, 1)
        k2 = self.k2.reshape(-1) if wall is None else torch.zeros(1, dtype=torch.float64, device=self.dev)
        if which == 0:
            A = lam * (d[:, 2] - k2 * d[:, 0]) - ni * (d[:, 3] - 2 * k2 * d[:, 2] + k2**2 * d[:, 0])
            g0, gn = st.w1[1], st.w1[2]  # no slip: dv/dy = 0
        else:
            A = lam * d[:, 0] - ni * (d[:, 2] - k2 * d[:, 0])
            g0, gn = st.d[1, 3], st.d[ny - 1, 3]  # no fourth derivative at the first and last rows
        # x(0) = x(ny) = 0; the ghost values follow from g0, gn
        c0, cn = [-g0[j] / g0[0] for j in (2, 3, 4)], [-gn[j] / gn[4] for j in (0, 1, 2)]
        A = A.clone()
        for j in range(3):
            A[0, 2 + j] += A[0, 0] * c0[j]
            A[-1, j] += A[-1, 4] * cn[j]
        x = _banded(A, b)
        zero = torch.zeros_like(x[0])
        lo = sum(c0[j] * x[j] for j in range(3))
        hi = sum(cn[j] * x[len(x) - 3 + j] for j in range(3))
        return torch.cat([lo[None], zero[None], x, zero[None], hi[None]])

    def start(self):
        self.dt = self.c["deltat"] or 1.0
        self.outstats(self.convolve(products=False)[1])

    def outstats(self, cfl):
        if self.c["cflmax"] > 0:
            self.dt = self.c["cflmax"] / cfl
        nz = self.c["nz"]
        U, W = self.V[0, :, 0, nz].real, self.V[2, :, 0, nz].real
        eu, ew = self.st.ends(self.st.w1, U), self.st.ends(self.st.w1, W)
        w = torch.as_tensor(self.st.wint, device=self.dev)
        return [self.time, float(eu[1]), -float(eu[2]), float(ew[1]), -float(ew[2]), float((w * U).sum()), self.px,
                float((w * W).sum()), 0.0, cfl * self.dt, self.dt]

    def step(self):
        st, ny, nz, ni = self.st, self.c["ny"], self.c["nz"], self.ni
        ta, tb, k2 = self.kx, self.kz, self.k2
        for o1, o2, o3 in RK:
            self.time += 2.0 / o1 * self.dt
            lam = o1 / self.dt
            (uu, vv, ww, uv, vw, uw), cfl = self.convolve()
            D = st.rows
            P = k2 * vv - ta * ta * uu - 2.0 * ta * tb * uw - tb * tb * ww
            Q = 1j * (ta * uv + tb * vw)
            ev = D(1, P) + D(2, Q) + k2 * D(0, Q)
            ee = D(0, ta * tb * (uu - ww) + (tb * tb - ta * ta) * uw) + D(1, 1j * (ta * vw - tb * uv))
            ee[:, 0, nz] = -(D(1, uv[:, 0, nz]).real + 1j * D(1, vw[:, 0, nz]).real)
            del uu, vv, ww, uv, vw, uw, P, Q
            v = self.V[1]
            s0, s2 = D(0, v), D(2, v)
            bv = lam * (s2 - k2 * s0) + ni * (D(3, v) - 2.0 * k2 * s2 + k2**2 * s0) + o2 * ev - o3 * self.old[1]
            eta = 1j * (tb * self.V[0] - ta * self.V[2])
            eta[:, 0, nz] = self.V[0, :, 0, nz].real + 1j * self.V[2, :, 0, nz].real
            s0 = D(0, eta)
            be = lam * s0 + ni * (D(2, eta) - k2 * s0) + o2 * ee - o3 * self.old[0]
            self.old = [ee, ev]
            del s0, s2, eta
            shape = (ny + 3,) + k2.shape
            v = self.solve(lam, bv.reshape(ny - 1, -1), 0).reshape(shape)
            eta = self.solve(lam, be.reshape(ny - 1, -1), 1).reshape(shape)
            del bv, be
            # the mean flow: the pressure gradient that gives the flow rate 4/3
            one = torch.ones((ny - 1, 1), dtype=torch.float64, device=self.dev)
            unit = self.solve(lam, one, 1, wall=True)[:, 0]
            w = torch.as_tensor(st.wint, device=self.dev)
            U, W = eta[:, 0, nz].real.clone(), eta[:, 0, nz].imag.clone()
            self.px = float((4.0 / 3.0 - (w * U).sum()) / (w * unit).sum())
            dv = st.derivative(v)
            q = k2.clone()
            q[0, nz] = 1.0
            self.V = torch.stack([1j * (ta * dv - tb * eta) / q, v, 1j * (tb * dv + ta * eta) / q])
            self.V[0, :, 0, nz] = (U + self.px * unit).to(torch.complex128)
            self.V[2, :, 0, nz] = W.to(torch.complex128)
        return self.outstats(cfl)

    def field(self):
        return self.V.permute(0, 2, 3, 1).contiguous()

    def budget(self, mean):
        """One sample of the Reynolds-stress budget spectra: (mean, spectra, profiles)."""
        c, st, nz, ny = self.c, self.st, self.c["nz"], self.c["ny"]
        U = torch.as_tensor(mean, device=self.dev)
        self.V[0, :, 0, nz] -= U
        G = self.gradient()
        N = [[], [], []]
        for s in self.chunks():
            u = [self.physical(F[s]) for F in self.V]
            for i in range(3):
                N[i].append(self.spectral(sum(self.physical(G[3 * i + k][s]) * u[k] for k in range(3))))
        N = [torch.cat(n) for n in N]
        wx = torch.full((c["nx"] + 1, 1), 2.0, dtype=torch.float64, device=self.dev)
        wx[0] = 1.0
        dot = lambda a, b: (wx * (a.conj() * b).real).sum(1)  # noqa: E731  (rows, kz)
        dU, dU2 = st.derivative(U), st.derivative(U, 2)
        Mj = [dU[:, None], 0.0, 0.0]  # dU_j/dy of the mean
        sp = torch.zeros((6, 10, 2 * nz + 1, ny + 3), dtype=torch.float64, device=self.dev)
        for r, (i, j) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (0, 2))):
            var = dot(self.V[i], self.V[j])
            prod = -(dot(self.V[i], self.V[1]) * Mj[j] + dot(self.V[j], self.V[1]) * Mj[i])
            diss = -2.0 * self.ni * sum(dot(G[3 * i + k], G[3 * j + k]) for k in range(3))
            turb = -dot(N[i], self.V[j]) - dot(N[j], self.V[i])
            for k, t in ((0, var), (1, prod), (2, diss), (3, turb), (4, self.ni * st.derivative(var, 2)),
                         (8, self.ni * st.derivative(var))):
                sp[r, k] = t.T
        m7 = torch.zeros((7, ny + 3), dtype=torch.float64, device=self.dev)
        m7[0], m7[2], m7[4] = U, dU, dU2
        return m7, sp, sp.sum(2)


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "ensemble":
            fields, lines = [], []
            for i, c in enumerate(_members(case, seed)):
                e = _Exact(c, seed + i)
                e.start()
                for _ in range(c["steps"]):
                    line = e.step()
                fields.append(e.field().reshape(-1).cpu())
                lines.append(line)
            return [torch.cat(fields).numpy(), np.array(lines)]
        e = _Exact(case, seed)
        if case["kind"] == "budget":
            return [x.cpu().numpy() for x in e.budget(_modes(case, seed)[0, 0, min(32, case["nz"])].real)]
        if case["kind"] == "closure":
            e.net = _network(seed)
        e.start()
        lines = [e.step() for _ in range(case["steps"])]
        return [e.field().cpu().numpy(), np.array(lines)]
