"""The rounding error of the explicit terms of `buildrhs` (dnsdata.f90:636-654)
in the FP64 and double-float paths: no larger than that of a plain evaluation,
stencil by stencil, in the same number format.

With ode = (0, 1, 0) and a vanishing viscosity the right-hand sides that
`buildrhs` leaves in the field are the explicit terms alone,

    v:   D1 P + (D2 + k2 D0) Q      eta:   D0 R + D1 S

of combinations P, Q, R, S of the six product spectra, linear in the stencils'
coefficients.  The handle's coefficients may differ from the oracle's in their
last bits; so, row by row, what a change of the 15 (10) coefficients can
explain is fitted over all modes and taken out of the difference from the
long-double evaluation.  What is left is rounding.

The bar is the same quantity for numpy's evaluation of the reference's stencils
in FP64; in double-float 2^5 times that, its unit being 2^-48 for 2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def field(p, seed):
    """A profile and perturbations of every mode that are smooth in y and fall with the wavenumber."""
    r = np.random.default_rng([seed, p.nx, p.nz])
    y = np.tanh(p.a * (2.0 * np.arange(-1, p.ny + 2) / p.ny - 1.0)) / np.tanh(p.a) + 1.0
    base = y * (2.0 - y)
    shape = (3, p.nx + 1, 2 * p.nz + 1, 3)
    c = r.standard_normal(shape) + 1j * r.standard_normal(shape)
    k2 = np.arange(p.nx + 1)[:, None] ** 2 + np.arange(-p.nz, p.nz + 1)[None, :] ** 2
    V = (c @ np.array([base, base * y, base**2])) * (0.03 * (1.0 + k2 / 4.0) ** -1.25)[None, :, :, None]
    V[:, 0, : p.nz] = np.conj(V[:, 0, : p.nz : -1])
    V[:, 0, p.nz] = V[:, 0, p.nz].real
    V[0, 0, p.nz] += base
    return V


def split(z):
    """Real and imaginary parts, modes and parts first, planes last."""
    z = z.reshape(-1, z.shape[-1])
    return np.concatenate([z.real, z.imag])


def combinations(p, VV, dtype):
    """P, Q, R, S of the products (6, nx+1, 2nz+1, planes) as real arrays (2 modes, planes), and k2 per row."""
    a = (LD(p.alfa0) * np.arange(p.nx + 1))[:, None, None]
    b = (LD(p.beta0) * np.arange(-p.nz, p.nz + 1))[None, :, None]
    uu, vv, ww, uv, vw, uw = VV.astype(dtype)
    P = (a * a + b * b) * vv - a * a * uu - 2 * a * b * uw - b * b * ww
    Q = 1j * (a * uv + b * vw)
    R = a * b * (uu - ww) + (b * b - a * a) * uw
    S = 1j * (a * vw - b * uv)
    S[0, p.nz] = -uv[0, p.nz].real - 1j * vw[0, p.nz].real
    k2 = np.broadcast_to(a * a + b * b, uu.shape[:2] + (1,)).reshape(-1)
    return [split(x) for x in (P, Q, R, S)], np.concatenate([k2, k2])[:, None]


def plain(p, VV, der):
    """numpy's FP64 evaluation of the reference's stencils (dnsdata.f90:636-654)."""
    a = (p.alfa0 * np.arange(p.nx + 1))[:, None, None]
    b = (p.beta0 * np.arange(-p.nz, p.nz + 1))[None, :, None]
    k2 = a * a + b * b
    n = p.ny - 1

    # planes are iy + 1: row iy reads planes iy-1 ... iy+3
    def DD(k, f):
        s = der[:, k, 0] * VV[f][..., 0:n]
        for j in range(1, 5):
            s = s + der[:, k, j] * VV[f][..., j : n + j]
        return s

    rhsu = -1j * a * DD(0, 0) - DD(1, 3) - 1j * b * DD(0, 5)
    rhsv = -1j * a * DD(0, 3) - DD(1, 1) - 1j * b * DD(0, 4)
    rhsw = -1j * a * DD(0, 5) - DD(1, 4) - 1j * b * DD(0, 2)
    ev = (1j * a * (1j * a * DD(1, 0) + DD(2, 3) + 1j * b * DD(1, 5))
          + 1j * b * (1j * a * DD(1, 5) + DD(2, 4) + 1j * b * DD(1, 2)) - k2 * rhsv)
    ee = 1j * b * rhsu - 1j * a * rhsw
    ee[0, p.nz] = rhsu[0, p.nz].real + 1j * rhsw[0, p.nz].real
    return ev, ee


def rounding(E, terms, der, n):
    """Relative rounding error of E (2 modes, rows) = sum over (stencil k, weights, F) of weights D_k F."""
    total = size = 0.0
    for i in range(n):
        exact = 0
        cols = []
        for k, w, F in terms:
            x = w * F[:, i : i + 5]
            exact = exact + x @ der[i, k].astype(LD)
            cols.append(x)
        e = (E[:, i].astype(LD) - exact).astype(np.float64)
        A = np.concatenate(cols, axis=1).astype(np.float64)
        A = A / np.maximum(np.linalg.norm(A, axis=0), 1e-300)
        e -= A @ np.linalg.lstsq(A, e, rcond=None)[0]
        total += float(e @ e)
        size += float((exact * exact).sum())
    return (total / size) ** 0.5


@pytest.mark.parametrize("prec,unit", [("fp64", 1.0), ("fp64dd", 32.0)])
@pytest.mark.parametrize("nx,ny,nz", [(20, 48, 17), (15, 101, 16), (9, 192, 12)])
def test_explicit_terms_round_no_worse_than_the_reference_stencils(gpu_lib, nx, ny, nz, prec, unit):
    import pyoracle
    from channel_gb300 import Channel, DnsIn

    p = DnsIn(nx=nx, ny=ny, nz=nz, alfa0=0.7, beta0=1.5, re=1e30, a=1.6, ymin=0.0, ymax=2.0, meanflowx=4.0 / 3.0,
              deltat=0.001, cflmax=0.0, nstep=1)
    with Channel(p, prec) as g:
        g.upload(field(p, 1))
        VV = g.products()
        g.buildrhs((0.0, 1.0, 0.0), False)
        G = g.download()[:2, :, :, 2:-2]
    der = pyoracle.Oracle(p).tables()["der"]
    (P, Q, R, S), k2 = combinations(p, VV, np.clongdouble)
    ev, ee = plain(p, VV, der)
    n = ny - 1
    for got, ref, terms in ((G[1], ev, ((1, 1, P), (2, 1, Q), (0, k2, Q))), (G[0], ee, ((0, 1, R), (1, 1, S)))):
        err, bar = rounding(split(got), terms, der, n), rounding(split(ref), terms, der, n)
        assert err <= unit * bar, (err, bar)


@pytest.mark.parametrize("prec", ["fp64", "fp64dd", "mixed"])
@pytest.mark.parametrize("nx,ny,nz", [(32, 48, 16), (24, 64, 24), (40, 96, 20)])
def test_rows_per_thread_do_not_change_the_results(gpu_lib, nx, ny, nz, prec):
    """The step in two halves runs k_rhs on half the modes and so with other rows per thread: the same bits, also at
    wavenumbers whose squares and products are rounded."""
    from channel_gb300 import Channel, DnsIn

    p = DnsIn(nx=nx, ny=ny, nz=nz, alfa0=1.1234567, beta0=3.0987, re=2000.0, a=1.6, ymin=0.0, ymax=2.0,
              meanflowx=4.0 / 3.0, deltat=0.002, cflmax=0.0, nstep=1)
    out = []
    for halves in (1, 2):
        with Channel(p, prec) as g:
            g.set_step_halves(halves)
            g.upload(field(p, 2))
            g.start()
            for _ in range(2):
                line = g.step()
            out.append((g.download(), line))
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
