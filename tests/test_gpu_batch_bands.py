"""Batches large enough for the batched band kernels: every grid equals its own
single-grid run bit for bit, with odd extents, grids without CPML and without z
faces between the others (no band blocks), sources on z-slab nodes, a Drude box,
and more grids than the band kernels' block has threads."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

NAMES = ("ex", "ey", "ez", "hx", "hy", "hz")


def _solver(shape, npml, faces, seed, drude=False):
    import fdtd_accelerate_gb300 as F
    rng = np.random.default_rng(seed)
    t = np.arange(12, dtype=np.float64)
    nx, ny, nz = shape
    src = [("ez", (nx // 2, ny // 2, nz // 2), np.sin(0.3 * t)), ("ex", (nx // 3, 8 % ny, 1), np.cos(0.2 * t)),
           ("ey", (nx // 3, ny // 2, nz - 2), np.sin(0.4 * t))]
    extra = {}
    if drude:
        extra["drude"] = F.DrudeAde(shape, (3, 4, 5), (9, 10, nz - 9))
        extra["drude"].set_coeff(0.2, 0.05)
    s = F.YeeSolver(shape, ce=[(0.5 / rng.uniform(1.0, 6.0, shape)).astype(np.float32) for _ in range(3)], npml=npml,
                    faces=faces, sources=src, **extra)
    s.set_fields(**{k: (0.1 * rng.standard_normal(shape)).astype(np.float32) for k in NAMES})
    return s


def _grids(kind):
    if kind == "many":  # 270 grids, 1.6 Mcells
        return [((18 + n % 3, 17, 19), 4 if n % 4 else 0, 0x3F, False) for n in range(270)]
    big = [((96, 80, 96), 8, 0x3F, False), ((30, 40, 44), 0, 0x3F, False), ((61, 97, 75), (5, 4, 9), 0x2A, False),
           ((50, 44, 70), 6, 0x0F, False), ((64, 64, 64), 8, 0x3F, kind == "drude"), ((20, 70, 33), 4, 0x3F, False)]
    return big


@pytest.mark.parametrize("kind", ["ragged", "drude", "many"])
@pytest.mark.parametrize("tile", [None, (16, 12, 1, 3)])
def test_batched_bands_bit_identical_to_single(kind, tile):
    import fdtd_accelerate_gb300 as F
    if kind == "many" and tile:
        pytest.skip("one launch shape is enough for many grids")
    cases = _grids(kind)
    assert sum(int(np.prod(c[0])) for c in cases) >= 3 << 19
    single = [_solver(sh, P, f, 50 + n, d) for n, (sh, P, f, d) in enumerate(cases)]
    batch = F.BatchSolver([_solver(sh, P, f, 50 + n, d) for n, (sh, P, f, d) in enumerate(cases)], tile=tile)
    for s in single:
        s.step(5)
    batch.step(2)
    batch.step(3)
    torch.cuda.synchronize()
    batch.check_status()
    for n, (a, b) in enumerate(zip(single, batch.solvers)):
        for k in NAMES:
            assert torch.equal(a.fields[k], b.fields[k]), (n, k)
        for q in range(6):
            if a.psi_e()[q] is not None:
                assert torch.equal(a.psi_e()[q], b.psi_e()[q]), (n, q)
                assert torch.equal(a.cpml.psi_h[q], b.cpml.psi_h[q]), (n, q)
