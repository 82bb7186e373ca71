"""The fixed-point transforms of the FP64 and double-float paths: the product
spectra of a plane against long-double transforms, for every padded length
that has a compile-time plan and for a length that has none; exact scaling by
powers of two; zeros; non-finite input.

Tolerances (relative L2 of a product's spectrum).  FP64: three roundings to
FP64 on the way (after the z-inverse, where they enter both factors, the x
pass and the z-forward), each 2^-53 / sqrt(3) rms = 6.4e-17, and as much again
from the fixed-point passes: 2.5e-16, times 4.  Double-float: the same with
2^-48, 2.1e-15 each: 8e-15, times 4.  White spectra, whose l1 norm is sqrt(N)
times their l2 norm, cost up to log2(sqrt(N)) more bits, of which the word's
nine spare bits leave at most three at the longest lengths: times 8.  (On
GB300 the FP64 products are off by 1.0-1.9e-16 on falling spectra and up to
4.4e-16 on white ones; FP64-pipe transforms by 3.1-4.9e-16 and 3.7-6.8e-16.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-15, "fp64dd": 3.2e-14}


def products_reference(S, nxd, nzd):
    """Product spectra of one plane's velocity spectra (3, nx+1, 2nz+1) in long double."""
    nx, nz = S.shape[1] - 1, S.shape[2] // 2
    Z = np.zeros((3, nx + 1, nzd), np.clongdouble)
    Z[:, :, : nz + 1], Z[:, :, nzd - nz:] = S[:, :, nz:], S[:, :, :nz]
    X = np.zeros((3, nxd + 1, nzd), np.clongdouble)
    X[:, : nx + 1] = np.fft.ifft(Z, axis=2) * np.longdouble(nzd)
    X[:, 0] = X[:, 0].real
    u, v, w = np.fft.irfft(X, n=2 * nxd, axis=1) * np.longdouble(2 * nxd)
    out = []
    for p in (u * u, v * v, w * w, u * v, v * w, u * w):
        Q = np.fft.fft(np.fft.rfft(p, axis=0)[: nx + 1], axis=1) / (np.longdouble(2 * nxd) * nzd)
        out.append(np.concatenate([Q[:, nzd - nz:], Q[:, : nz + 1]], axis=1))
    return np.array(out)


def channel(nx, nz, prec):
    from channel_gb300 import Channel, DnsIn

    p = DnsIn(nx=nx, ny=10, nz=nz, alfa0=1.0, beta0=2.0, re=2000.0, a=1.5, ymin=0.0, ymax=2.0, meanflowx=4.0 / 3.0,
              deltat=0.001, cflmax=0.0, nstep=1)
    return p, Channel(p, prec)


def spectrum(p, kind, seed=0):
    """A real field's spectra on every plane: white, or falling with the wavenumber under a mean profile."""
    r = np.random.default_rng([seed, p.nx, p.nz])
    V = r.standard_normal((3, p.nx + 1, 2 * p.nz + 1, p.ny + 3)) + 1j * r.standard_normal((3, p.nx + 1, 2 * p.nz + 1, p.ny + 3))
    if kind == "steep":
        k2 = np.arange(p.nx + 1)[:, None] ** 2 + np.arange(-p.nz, p.nz + 1)[None, :] ** 2
        V *= 0.03 * (1.0 + k2 / 4.0)[None, :, :, None] ** -1.25
    V[:, 0, :p.nz] = np.conj(V[:, 0, :p.nz:-1])
    V[:, 0, p.nz] = V[:, 0, p.nz].real
    if kind == "steep":
        V[0, 0, p.nz] = 1.0
    return V


# (nx, nz) of every planned x length 32 ... 768 and z length 32 ... 1536, at the smallest or largest mode
# count of the length, and one without a plan
SIZES = [(16, 10), (31, 16), (42, 21), (63, 32), (64, 42), (127, 64), (128, 85), (171, 86), (256, 129), (342, 171),
         (16, 257), (16, 511), (7, 4)]


@pytest.mark.parametrize("prec", ["fp64", "fp64dd"])
@pytest.mark.parametrize("nx,nz", SIZES)
def test_products_against_long_double(gpu_lib, nx, nz, prec):
    p, g = channel(nx, nz, prec)
    with g:
        for kind, tol in (("steep", TOL[prec]), ("white", 8 * TOL[prec])):
            V = spectrum(p, kind)
            g.upload(V)
            P = g.products()
            plane = 5
            R = products_reference(V[..., plane], p.nxd, p.nzd)
            for k in range(6):
                err = np.linalg.norm((P[k, :, :, plane] - R[k]).ravel()) / np.linalg.norm(R[k].ravel())
                assert err <= tol, (kind, k, float(err))


@pytest.mark.parametrize("prec,shift", [("fp64", 150), ("fp64", -150), ("fp64dd", 20), ("fp64dd", -20)])
def test_scaling_is_exact(gpu_lib, prec, shift):
    """Columns and rows carry their own exponents: a field times a power of two gives the same bits, shifted."""
    p, g = channel(42, 32, prec)
    with g:
        V = spectrum(p, "steep")
        g.upload(V)
        P = g.products()
        g.upload(V * 2.0**shift)
        assert np.array_equal(g.products(), P * 2.0 ** (2 * shift))


@pytest.mark.parametrize("prec", ["fp64", "fp64dd"])
def test_zeros_and_small_columns(gpu_lib, prec):
    p, g = channel(42, 32, prec)
    with g:
        V = np.zeros((3, p.nx + 1, 2 * p.nz + 1, p.ny + 3), complex)
        g.upload(V)
        assert not g.products().any()
        V[0, 0, p.nz] = 1.0
        V[2, 3, p.nz + 5] = 1e-15  # far below u, and products with v = 0 stay zero
        g.upload(V)
        P = g.products()
        assert not P[[1, 3, 4]].any()
        np.testing.assert_allclose(P[5, 3, p.nz + 5].real, 1e-15, rtol=1e-12)
        np.testing.assert_allclose(P[0, 0, p.nz].real, 1.0, rtol=1e-14)


@pytest.mark.parametrize("prec", ["fp64", "fp64dd"])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_non_finite_is_reported(gpu_lib, prec, value):
    from channel_gb300.lib import ChannelError

    p, g = channel(42, 32, prec)
    with g:
        V = spectrum(p, "steep")
        V[1, 2, 3, 6] = value
        g.upload(V)
        with pytest.raises(ChannelError, match="non-finite"):
            g.start()
