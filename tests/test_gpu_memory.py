"""Device memory that a handle can do without is given up before a call is
refused: the factors of the second and third substeps, two thirds of the
factors' memory, are kept only by the solve forms that use them, and neither the
creation of a handle nor a later allocation of its own fails for them.

The rest of the device's memory is taken by a plain allocation meanwhile; the
bounds come from the handle's own use, measured with memory to spare."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def params(nx, ny, nz):
    from channel_gb300 import DnsIn

    return DnsIn(nx=nx, ny=ny, nz=nz, alfa0=1.0, beta0=2.0, re=3000.0, a=1.6, ymin=0.0, ymax=2.0,
                 meanflowx=4.0 / 3.0, deltat=0.001, cflmax=0.0, nstep=1)


def rest(p):
    """Bytes of the factors of two substeps."""
    return 2 * 10 * 8 * (p.ny - 1) * (p.nx + 1) * (p.nz + 1)


def free():
    import torch

    return torch.cuda.mem_get_info()[0]


def leave(nbytes):
    """An allocation that leaves about that many bytes free."""
    import torch

    torch.cuda.empty_cache()
    return torch.empty(free() - nbytes, dtype=torch.uint8, device="cuda")


@pytest.fixture(autouse=True)
def no_cache(gpu_lib):
    torch = pytest.importorskip("torch")
    yield
    torch.cuda.empty_cache()


def steps(p, V0, tiles=None):
    from channel_gb300 import Channel

    with Channel(p, "fp64") as g:
        if tiles:
            g.set_tiles(g.tiles()[:5] + tiles)
        g.upload(V0)
        g.start()
        for _ in range(2):
            line = g.step()
        return g.download(), line


def test_forms_that_need_one_set_of_factors_keep_one(gpu_lib):
    from channel_gb300 import Channel, initial

    p = params(63, 96, 63)
    ref = steps(p, initial.perturbed_laminar(p, 0.01, 1))
    with Channel(p, "fp64") as g:
        base = g.tiles()
        assert base[5] >= 3  # the default form here factors ahead
        with_rest = free()
        g.set_tiles(base[:5] + (1, 1))
        assert free() - with_rest >= 0.9 * rest(p)
        g.set_tiles(base)
        assert free() - with_rest <= 0.1 * rest(p)
    for form in (1, 2, 3, 4, 5):
        V, line = steps(p, initial.perturbed_laminar(p, 0.01, 1), (form, 1))
        assert np.array_equal(V, ref[0]) and np.array_equal(line, ref[1])


def test_handle_without_room_for_the_rest(gpu_lib):
    """A handle whose other buffers just fit is made, and steps alike."""
    from channel_gb300 import Channel, initial

    p = params(127, 96, 127)
    V0 = initial.perturbed_laminar(p, 0.01, 1)
    ref = steps(p, V0)
    before = free()
    with Channel(p, "fp64"):
        used = before - free()
    hog = leave(used - rest(p) // 2)
    try:
        V, line = steps(p, V0)
    finally:
        del hog
    assert np.array_equal(V, ref[0]) and np.array_equal(line, ref[1])


def test_later_allocation_takes_the_rest_back(gpu_lib):
    """The budget spectra's buffers of a handle that has all its factors, with too little memory left for both."""
    from channel_gb300 import Channel, initial

    p = params(127, 96, 127)
    V0 = initial.perturbed_laminar(p, 0.01, 1)
    mean = V0[0, 0, p.nz].real.copy()
    out = []
    for short in (False, True):
        with Channel(p, "fp64") as g:
            g.upload(V0)
            g.start()
            g.step()
            before = free()
            hog = leave(need - rest(p) // 2) if short else None
            try:
                g.tke_reset(mean, np.zeros_like(mean))
                if not short:
                    need = before - free()
                g.step()
                g.tke_accumulate()
                out.append([g.download()] + list(g.tke_result()[:3]))
            finally:
                del hog
    for a, b in zip(*out):
        assert np.array_equal(a, b)
