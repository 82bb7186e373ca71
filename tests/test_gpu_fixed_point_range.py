"""The fixed-point transforms at the ends of their range: data near the largest
and smallest numbers of the type, and spectra that come closest to the bounds
from which the headroom of the passes is derived - all modes in phase at 45
degrees, signs that alternate, and single modes at every residue of the first
pass, whose values have |re| = |im| at the bound of the modulus - for every
planned length, against long double.

Tolerances (relative L2): single modes as falling spectra in
test_gpu_fixed_point.py; a coherent spectrum's products are flat, and FP64
transforms are off by at most 4.5e-16 of them at these lengths: 5e-16 in FP64.
Powers of two: the bits of the unscaled run where every column's values reach
2^-959.  Below that one unit is the smallest normal number: after the x rows
an error of one unit for each of nzd values of a column and again in its
transform.  Double-float spectra: half a smallest subnormal in either float."""
import numpy as np
import pytest
from test_gpu_fixed_point import SIZES, TOL, channel, products_reference, spectrum

pytestmark = pytest.mark.gpu

COHERENT = {"fp64": 5e-16, "fp64dd": TOL["fp64dd"]}


@pytest.mark.parametrize("prec,shift", [("fp64", 440), ("fp64", 500), ("fp64", -450), ("fp64", -505), ("fp64dd", 55),
                                        ("fp64dd", -55), ("fp64dd", -62)])
@pytest.mark.parametrize("nx,nz", [(42, 32), (20, 40)])
def test_products_up_to_the_ends_of_the_range(gpu_lib, prec, shift, nx, nz):
    p, g = channel(nx, nz, prec)
    with g:
        V = spectrum(p, "steep")
        g.upload(V)
        P = g.products()
        g.upload(V * 2.0**shift)
        Q = g.products()
    assert np.isfinite(Q.view(float)).all()
    tol = {("fp64", -505): 2 * p.nzd * 2.0**-1022, ("fp64dd", -55): 2.0**-149, ("fp64dd", -62): 2.0**-149}.get((prec, shift), 0.0)
    D = Q * 2.0**-shift * 2.0**-shift - P
    assert np.abs(D.view(float)).max() <= tol * 2.0**-shift * 2.0**-shift


@pytest.mark.parametrize("shift", [960, 900, -900])
def test_cfl_up_to_the_ends_of_the_range(gpu_lib, shift):
    p, g = channel(42, 32, "fp64")
    with g:
        V = spectrum(p, "steep")
        g.upload(V)
        cfl = g.start()[9]
        g.upload(V * 2.0**shift)
        assert g.start()[9] == cfl * 2.0**shift


def coherent(p, kind):
    """All modes in phase at 45 degrees; `alternating`: with signs that move the peak to the middle."""
    nx, nz = p.nx, p.nz
    s = np.ones((nx + 1, 2 * nz + 1))
    if kind == "alternating":
        s = (-1.0) ** (np.arange(nx + 1)[:, None] + np.arange(-nz, nz + 1)[None, :])
    V = (1 + 1j) * s
    V[0, :nz] = np.conj(V[0, :nz:-1])
    V[0, nz] = V[0, nz].real
    return np.broadcast_to(V * np.array([1.0, 0.75, 0.3])[:, None, None], (3, nx + 1, 2 * nz + 1))


@pytest.mark.parametrize("prec", ["fp64", "fp64dd"])
@pytest.mark.parametrize("nx,nz", SIZES)
def test_coherent_spectra(gpu_lib, nx, nz, prec):
    p, g = channel(nx, nz, prec)
    kinds = ("in phase", "alternating")
    with g:
        V = np.zeros((3, nx + 1, 2 * nz + 1, p.ny + 3), complex)
        for i, kind in enumerate(kinds):
            V[..., i] = coherent(p, kind)
        g.upload(V)
        P = g.products()
    for i, kind in enumerate(kinds):
        R = products_reference(V[..., i], p.nxd, p.nzd)
        for k in range(6):
            err = np.linalg.norm((P[k, :, :, i] - R[k]).ravel()) / np.linalg.norm(R[k].ravel())
            assert err <= COHERENT[prec], (kind, k, float(err))


@pytest.mark.parametrize("prec", ["fp64", "fp64dd"])
@pytest.mark.parametrize("nx,nz", SIZES)
def test_single_modes(gpu_lib, nx, nz, prec):
    """u = v = w = a e^{i(kx x + kz z)} + c.c., kx > 0: every product is 2 |a|^2 at (0, 0) and a^2 at (2 kx,
    2 kz)."""
    p, g = channel(nx, nz, prec)
    a = 0.75 * (1 - 1j)
    with g:
        planes = p.ny + 3
        modes = [(1 + q % nx, (q * 7) % (2 * nz + 1) - nz) for q in range(3 * planes)]
        for first in range(0, len(modes), planes):
            V = np.zeros((3, nx + 1, 2 * nz + 1, planes), complex)
            R = np.zeros((nx + 1, 2 * nz + 1, planes), complex)
            for i, (kx, kz) in enumerate(modes[first : first + planes]):
                V[:, kx, nz + kz, i] = a
                R[0, nz, i] = 2 * abs(a) ** 2
                kz2 = (2 * kz + nz) % p.nzd - nz  # nzd = 3 nz: 2 nz is seen at -nz
                if 2 * kx <= nx and kz2 <= nz:
                    R[2 * kx, nz + kz2, i] = a * a
            g.upload(V)
            P = g.products()
            err = np.linalg.norm((P - R).reshape(6, -1, planes), axis=1) / np.linalg.norm(R.reshape(-1, planes), axis=0)
            assert err.max() <= TOL[prec], float(err.max())
