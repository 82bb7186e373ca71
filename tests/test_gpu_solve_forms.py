"""The solve forms against each other, bit for bit, where their block shapes
change: eight threads per pair in four parts up to two blocks of 16 pairs on
each SM and in two parts beyond, in every precision (double-float recovers u
and w by its own code), with a time step that changes from step to step, so that
the factors of all three substeps, made at the step's start, are those of the
new step; and the default form against the oracle on both sides of the line.

Tolerance of the oracle comparison: the parity tests' one-step bar, 1e-12
relative L2 per velocity component."""
import numpy as np
import pytest

from helpers import per_field_rel

pytestmark = pytest.mark.gpu


def params(nx, ny, nz, adaptive):
    from channel_gb300 import DnsIn

    return DnsIn(nx=nx, ny=ny, nz=nz, alfa0=1.1, beta0=2.3, re=3000.0, a=1.6, ymin=0.0, ymax=2.0, meanflowx=4.0 / 3.0,
                 deltat=0.0 if adaptive else 0.002, cflmax=0.8 if adaptive else 0.0, nstep=4)


def edge():
    """nz with exactly two blocks of 16 pairs per SM at nx = 63, and one more pair row."""
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return sms * 32 // 64 - 1


# pairs below, at and above the line between four and two parts
@pytest.mark.parametrize("prec", ["fp64", "fp64dd", "mixed"])
@pytest.mark.parametrize("nx,ny,nz", [(20, 33, 19), (63, 12, None), (63, 12, "next"), (79, 20, 75)])
def test_forms_are_identical(gpu_lib, nx, ny, nz, prec):
    from channel_gb300 import Channel, initial

    pytest.importorskip("torch")
    nz = edge() if nz is None else edge() + 1 if nz == "next" else nz
    p = params(nx, ny, nz, True)
    V0 = initial.perturbed_laminar(p, 0.02, 6)
    out = []
    for form in (1, 2, 3, 4, 5):
        for halves in (1, 2):
            with Channel(p, prec) as g:
                g.set_tiles(g.tiles()[:5] + (form, halves))
                g.upload(V0)
                g.start()
                lines = [g.step() for _ in range(3)]
                out.append((g.download(), np.array(lines)))
    dt = out[0][1][:, 10]
    assert len(set(dt)) >= 2  # the step did change
    for V, lines in out[1:]:
        assert np.array_equal(V, out[0][0])
        assert np.array_equal(lines, out[0][1])


@pytest.mark.parametrize("prec", ["fp64", "fp64dd"])
@pytest.mark.parametrize("nx,ny,nz", [(63, 16, 63), (79, 20, 75), (99, 12, 99)])
def test_default_form_matches_oracle(gpu_lib, nx, ny, nz, prec):
    import pyoracle
    from channel_gb300 import Channel, initial

    p = params(nx, ny, nz, False)
    V0 = initial.perturbed_laminar(p, 0.02, 3)
    o = pyoracle.Oracle(p)
    o.set_field(V0)
    o.start()
    with Channel(p, prec) as g:
        g.upload(V0)
        g.start()
        for _ in range(2):
            o.step()
            g.step()
        e = per_field_rel(g.download(), o.field())
    assert max(e) <= 1e-12, e
