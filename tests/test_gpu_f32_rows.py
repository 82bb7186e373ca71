"""The FP32 transforms of the mixed step: the product spectra of a plane
against long-double transforms for every x length with a compile-time plan, at
mode counts on both sides of half a row (the row is unpacked two modes at a
time), with the registers of three and of four resident blocks.

Tolerance (relative L2 of a product's spectrum): 2 (log2 nxd + log2 nzd) < 40
butterfly levels, each rounding twice (twiddle and sum) at 2^-24 / sqrt(3) =
3.4e-8 rms, in both factors: sqrt(40 * 2 * 2) * 3.4e-8 = 4.3e-7, times 4."""
import numpy as np
import pytest

from test_gpu_fixed_point import channel, products_reference, spectrum

pytestmark = pytest.mark.gpu

TOL = 1.7e-6


@pytest.mark.parametrize("nx,nxd", [(16, 32), (20, 32), (21, 48), (31, 48), (33, 64), (42, 64), (43, 96), (48, 96),
                                    (63, 96), (86, 192), (96, 192), (127, 192), (200, 384), (255, 384), (342, 768),
                                    (384, 768), (400, 768)])
def test_products_against_long_double(gpu_lib, nx, nxd):
    p, g = channel(nx, 13, "mixed")
    with g:
        V = spectrum(p, "steep")
        plane = 5
        R = products_reference(V[..., plane], p.nxd, p.nzd)
        t, got = g.tiles(), []
        assert t[2] >= 4 and p.nxd == nxd
        for variant in (4, 5):
            g.set_tiles(t[:2] + (variant,) + t[3:])
            g.upload(V)
            got.append(g.products()[..., plane])
        assert np.array_equal(got[0], got[1])
        for k in range(6):
            err = np.linalg.norm((got[0][k] - R[k]).ravel()) / np.linalg.norm(R[k].ravel())
            assert err <= TOL, (k, float(err))
