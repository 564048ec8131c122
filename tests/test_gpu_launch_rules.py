"""Launch rules of the fused step on the forms that an earlier rule slowed down: the
route taken, and the step through it equal to the array calls bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

NAMES = ("ex", "ey", "ez", "hx", "hy", "hz")


def solver(shape, npml, drude=False, tfsf=False, tile=None):
    import fdtd_accelerate_gb300 as F
    rng = np.random.default_rng(8)
    extra = {}
    if drude:
        extra["drude"] = F.DrudeAde(shape, [n // 4 for n in shape], [n // 2 for n in shape])
        extra["drude"].set_coeff(0.2, 0.05)
    if tfsf:
        extra["tfsf"] = F.Tfsf(shape, [npml + 5] * 3, [n - npml - 6 for n in shape], wavelength=12.0, steps=16)
    s = F.YeeSolver(shape, npml=npml, tile=tile, sources=[("ez", tuple(n // 2 for n in shape), np.sin(0.3 * np.arange(12.0)))],
                    **extra)
    s.set_fields(**{k: (0.1 * rng.standard_normal(shape)).astype(np.float32) for k in NAMES})
    return s


def check(a, b, n=3):
    a.step(n)
    b.step_unfused(n)
    torch.cuda.synchronize()
    a.check_status()
    for k in NAMES:
        assert torch.equal(a.fields[k], b.fields[k]), k
    for q in range(6):
        if a.psi_e()[q] is not None:
            assert torch.equal(a.psi_e()[q], b.psi_e()[q]) and torch.equal(a.cpml.psi_h[q], b.cpml.psi_h[q]), q


@pytest.mark.parametrize("shape,npml,drude,band", [
    ((1000, 60, 20), 8, False, 1),     # rows that are mostly slab
    ((197, 200, 20), 8, True, 1),      # the line of such rows: 786432 cells
    ((196, 200, 20), 8, True, 0),
    ((52, 162, 171), 8, True, 1),
    ((95, 95, 95), 6, False, 1),       # the line of the others: 851968 cells
    ((94, 95, 95), 6, False, 0)])
def test_z_slab_route(shape, npml, drude, band):
    a, b = (solver(shape, npml, drude) for _ in range(2))
    assert a.plan_info()["z_band"] == band
    check(a, b)


@pytest.mark.parametrize("shape,drude,tfsf,tile,band", [
    ((80, 80, 80), True, True, (4,), 1), ((80, 80, 80), True, False, (4, 0, 0, 4), 1), ((80, 80, 80), True, True, None, 0),
    ((70, 72, 72), False, False, (4,), 0), ((80, 80, 80), False, False, (4,), 1), ((64, 64, 64), True, True, (4, 0, 0, 6), 0),
    ((48, 48, 48), False, True, (8, 8), 1), ((64, 64, 64), False, False, (8, 31), 1), ((57, 100, 124), False, False, (8, 64), 1),
    ((48, 48, 48), False, False, (8, 48), 0), ((48, 48, 48), True, False, (8, 48), 1), ((64, 64, 64), False, False, (8, 7), 0)])
def test_z_slab_route_of_the_callers_launch_shapes(shape, drude, tfsf, tile, band):
    a, b = (solver(shape, 4, drude, tfsf, tile) for _ in range(2))
    assert a.plan_info()["z_band"] == band
    check(a, b)


@pytest.mark.parametrize("shape,npml,drude,tile,most", [
    ((180, 180, 180), 4, False, None, 16), ((300, 120, 120), 8, True, None, 16), ((125, 125, 130), 8, False, None, 8),
    ((125, 125, 130), 8, False, (8, 40), 40)])
def test_x_chunk_with_a_wave(shape, npml, drude, tile, most):
    """Grids with a wave and CPML whose launch would be one round of long items take
    chunks that give 3 items an SM; a chunk of the caller's stays."""
    a, b = (solver(shape, npml, drude, True, tile) for _ in range(2))
    assert a.plan_info()["x_chunk"] == most
    check(a, b)


@pytest.mark.parametrize("npml,drude,tile,launches", [(0, True, None, 1), (5, True, (4,), 3), (5, False, (4, 20, 0, 6), 3),
                                                      (5, True, None, 1)])
def test_batch_routes(npml, drude, tile, launches):
    """Small batches: band launches for tiles of 4 rows, none without a z layer."""
    import ctypes as C
    import fdtd_accelerate_gb300 as F
    from fdtd_accelerate_gb300 import _native as N
    shapes = [(24 + q, 30, 22 + 3 * q) for q in range(8)]
    a, b = ([solver(sh, npml, drude and q % 2 == 0) for q, sh in enumerate(shapes)] for _ in range(2))
    batch = F.BatchSolver(a, tile=tile)
    info = (C.c_int32 * 8)()
    N.call("fdtd_batch_plan_info", batch.plan(), info, 8)
    batch.step(1)
    batch.step(2)
    torch.cuda.synchronize()
    batch.check_status()
    for s, r in zip(a, b):
        r.step_unfused(3)
        for k in NAMES:
            assert torch.equal(s.fields[k], r.fields[k]), k
    assert info[7] == launches
