"""The fixed-point x rows beyond the plain products (tests/test_gpu_fixed_point.py):
with the closure's stresses, against the generic kernels, and those of the
budget spectra, against the oracle, over the planned x lengths.

Tolerance of the stresses (relative L2 of the right-hand sides): both sides'
product spectra are off by at most the tolerance of test_gpu_fixed_point, 1e-15
(FP64) and 3.2e-14 (double-float, whose generic transforms have its 48 bits),
and the right-hand sides take two y derivatives on ten points, whose stencils
amplify noise against the falling spectra by up to 100: 2e-13 and 6.4e-12."""
import numpy as np
import pytest

from test_gpu_fixed_point import channel, spectrum
from test_gpu_tke import run_case

pytestmark = pytest.mark.gpu

TOL = {"fp64": 2e-13, "fp64dd": 6.4e-12}


@pytest.mark.parametrize("prec", ["fp64", "fp64dd"])
@pytest.mark.parametrize("nx,nz", [(20, 10), (31, 16), (42, 21), (63, 32), (84, 42), (127, 12), (170, 10), (255, 8),
                                   (341, 12), (400, 8)])
def test_stresses_against_the_generic_rows(gpu_lib, nx, nz, prec):
    p, g = channel(nx, nz, prec)
    r = np.random.default_rng(nx)
    with g:
        t = g.tiles()
        assert t[2] >= 4
        # the field and the stresses of like size, either far larger, the field zero, the stresses zero
        for vs, ts in ((1.0, 1e-2), (1.0, 1e-12), (1e-6, 1.0), (0.0, 1.0), (1.0, 0.0)):
            V = vs * spectrum(p, "steep")
            g.closure_set_tau((ts * r.standard_normal((6, g.closure_points()))).astype(np.float32))
            out = []
            for tiles in (t, (1, 1, 2) + t[3:]):
                g.set_tiles(tiles)
                g.upload(V)
                g.start(deltat=1e-3)
                g.buildrhs((120.0 / 32.0, 2.0, 0.0), False)
                out.append(g.download())
            err = np.linalg.norm((out[0] - out[1]).ravel()) / np.linalg.norm(out[1].ravel())
            assert err <= TOL[prec], (vs, ts, float(err))


@pytest.mark.parametrize("nx,nz", [(20, 10), (31, 13), (42, 16), (63, 12), (84, 20), (127, 9), (170, 8), (255, 6),
                                   (341, 6), (400, 5)])
def test_budget_spectra(gpu_lib, nx, nz):
    from channel_gb300 import dnsin

    run_case(dnsin.DnsIn(nx=nx, ny=12, nz=nz, alfa0=1.3, beta0=2.1, re=3000.0, a=1.6, ymin=0.0, ymax=2.0,
                         meanflowx=4.0 / 3.0, deltat=0.001, cflmax=0.0, nstep=3), False, False)


def test_budget_spectra_of_a_mixed_handle(gpu_lib):
    """The budget kernels are the FP64 ones in every precision: the same field, the same bits."""
    out = []
    for prec in ("mixed", "fp64"):
        p, g = channel(42, 21, prec)
        with g:
            g.upload(spectrum(p, "steep"))
            U = np.linspace(0.0, 1.0, p.ny + 3)
            g.tke_reset(U, 0 * U)
            g.tke_accumulate()
            out.append(g.tke_result()[1])
    assert np.array_equal(out[0], out[1])
