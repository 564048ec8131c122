"""Fused step with the z-slab terms inside the kernel (grids of 2048 rows and
more outside the band kernels' range) and its edges: groups of 4 cells on nodes
of both z slabs, odd slab widths, rows that are no multiple of 4 floats, tile
rows with and without y slab cells, chunks of two planes, one x chunk.  Equal
bit for bit to the reference-shaped kernels, fields and psi."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

NAMES = ("ex", "ey", "ez", "hx", "hy", "hz")


def _pair(shape, npml, faces, tile=None, seed=3, **extra):
    import fdtd_accelerate_gb300 as F
    rng = np.random.default_rng(seed)
    ce = [(0.5 / rng.uniform(1.0, 6.0, shape)).astype(np.float32) for _ in range(3)]
    init = {k: (0.1 * rng.standard_normal(shape)).astype(np.float32) for k in NAMES}
    t = np.arange(12, dtype=np.float64)
    nx, ny, nz = shape
    src = [("ez", (nx // 2, ny // 2, nz // 2), F.gaussian_sine(t, 3.0, 2.0, 0.1)),
           ("ex", (nx // 3, 8 % ny, 1), F.gaussian_sine(t, 4.0, 2.0, 0.1)),
           ("ey", (nx // 3, 7, nz - 2), F.gaussian_sine(t, 2.0, 2.0, 0.1))]
    out = []
    for _ in range(2):
        s = F.YeeSolver(shape, ce=ce, npml=npml, faces=faces, sources=src, tile=tile,
                        **{k: v() for k, v in extra.items()})
        s.set_fields(**init)
        out.append(s)
    return out


def _check(a, b, n=6):
    a.step(n)
    b.step_unfused(n)
    torch.cuda.synchronize()
    a.check_status()
    for k in NAMES:
        assert torch.equal(a.fields[k], b.fields[k]), k
    for q in range(6):
        if a.psi_e()[q] is not None:
            assert torch.equal(a.psi_e()[q], b.psi_e()[q]), "psi_e%d" % q
            assert torch.equal(a.cpml.psi_h[q], b.cpml.psi_h[q]), "psi_h%d" % q


@pytest.mark.parametrize("shape,npml,faces,tile", [
    ((48, 48, 12), 5, 0x3F, None),             # nz = 2P+2: one group on nodes of both z slabs
    ((48, 48, 13), 5, 0x3F, None),
    ((46, 50, 15), 5, 0x30, None),
    ((48, 48, 66), 7, 0x3F, None),             # second z tile of two cells, odd slab width
    ((47, 45, 128), 12, 0x3F, None),           # one slab a z tile
    ((48, 44, 157), 10, 0x3F, (8, 48, 0, 3)),  # one x chunk, ragged rows
    ((50, 46, 80), (4, 6, 17), 0x3F, None),    # slab wider than 4 groups
    ((45, 47, 64), 8, 0x20, (16, 5, 0, 3)),
    ((45, 47, 70), 8, 0x1F, (4, 6, 2, 4)),     # persistent grid, no z back face
    ((64, 32, 72), 3, 0x0C, None),             # y faces alone
    ((161, 72, 70), 4, 0x3F, (8, 2, 0, 3)),    # 1458 items: clusters of 8, the last one not full
])
def test_z_terms_in_kernel(shape, npml, faces, tile):
    a, b = _pair(shape, npml, faces, tile)
    assert a.plan_info()["z_band"] == 0 and a.plan_info()["launches_per_step"] == 1
    _check(a, b)


@pytest.mark.parametrize("k0,nk", [(12, 16), (13, 17)])  # rows of the box: multiples of 4 cells, and not
def test_drude_and_tfsf_with_z_terms(k0, nk):
    import fdtd_accelerate_gb300 as F
    shape, npml = (48, 48, 44), 5

    def drude():
        d = F.DrudeAde(shape, (10, 12, k0), (20, 21, nk))
        d.set_coeff(0.2, 0.05)
        return d

    def tfsf():
        return F.Tfsf(shape, (9, 10, 9), (38, 36, 33), wavelength=12.0, propagation_direction=("normal", "y"),
                      polarization_angle=0.7, steps=16)

    for extra in ({"drude": drude}, {"tfsf": tfsf}, {"drude": drude, "tfsf": tfsf}):
        a, b = _pair(shape, npml, 0x3F, **extra)
        _check(a, b)
        if "drude" in extra:
            assert torch.equal(a.drude.J, b.drude.J)


def test_band_range_and_plain_chunks():
    """The band kernels' range (2^21 cells and more), and plain grids at sizes
    where the chunk rule gives several rounds, one round and one chunk."""
    a, b = _pair((128, 130, 127), 6, 0x3F)
    assert a.plan_info()["z_band"] == 1
    _check(a, b, 3)
    for shape in ((130, 96, 200), (33, 64, 64), (9, 8, 8), (2, 2, 2)):
        a, b = _pair(shape, 0, 0x3F) if min(shape) > 8 else (None, None)
        if a is None:
            import fdtd_accelerate_gb300 as F
            a, b = F.YeeSolver(shape), F.YeeSolver(shape)
            for s in (a, b):
                s.set_fields(**{k: np.random.default_rng(1).standard_normal(shape) for k in NAMES})
        _check(a, b, 4)


def _cluster(ranges, n, seed, ny=128, nz=128):
    """n sources in each x range, rows 9..14, columns 70..100 of one tile, and n/4 repeats."""
    rng = np.random.default_rng(seed)
    amp = rng.standard_normal((n, 8))
    src = []
    for x0, x1 in ranges:
        for m in range(n):
            at = (int(rng.integers(x0, x1)), int(rng.integers(9, 15)), int(rng.integers(70, 101)))
            src.append((("ex", "ey", "ez")[m % 3], at if m % 4 else (x0, 9, 70), amp[m]))
    return src


@pytest.mark.parametrize("batch", [False, True])
def test_sources_counted_per_default_chunk(batch):
    """Sources are counted against the capacity of an item in chunks of 8 planes on these
    grids (3 items an SM), not in the longer chunks the step takes: 120 in planes 1..6 and
    120 in 9..14 are accepted, and applied although they share an item; 129 in 1..6 are refused."""
    import fdtd_accelerate_gb300 as F
    shape = (96, 128, 128) if batch else (128, 128, 128)

    def build(src):
        s = [F.YeeSolver(shape, npml=6, sources=src) for _ in range(2)]
        for u in s:
            u.set_fields(**{k: np.random.default_rng(5).standard_normal(shape).astype(np.float32) for k in NAMES})
        if not batch:
            return s, s[0]
        return s, F.BatchSolver([s[0]] + [F.YeeSolver(shape, npml=6) for _ in range(7)])

    s, run = build(_cluster(((1, 7), (9, 15)), 120, 7))
    run.step(4)
    s[1].step_unfused(4)
    torch.cuda.synchronize()
    run.check_status()
    if not batch:
        assert run.plan_info()["x_chunk"] > 8
    for k in NAMES:
        assert torch.equal(s[0].fields[k], s[1].fields[k]), k
    with pytest.raises(ValueError):
        s, run = build(_cluster(((1, 7),), 129, 8))
        run.step(1)
