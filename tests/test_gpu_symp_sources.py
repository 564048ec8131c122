"""Sources of the 4th-order stage pairs: a long list on a grid that is all shell."""
import pytest
import torch

from tests.test_gpu_symp_layout import assert_same, coefs, solver

pytestmark = pytest.mark.gpu


def spread(shape, each):
    """`each` sources in every 16 x 32 tile, every fifth one a repeat of a cell before it."""
    out = []
    for j0 in range(0, shape[1], 16):
        for k0 in range(0, shape[2], 32):
            at = [("ex", "ey", "ez")[q % 3] for q in range(each)]
            ijk = [((7 * q) % shape[0], j0 + (3 * q) % 16, k0 + (5 * q) % 32) for q in range(each)]
            for q in range(4, each, 5):
                at[q], ijk[q] = at[q - 3], ijk[q - 3]
            out += [(c, x, lambda t, q=q: 1e-4 * (q + 1) * t) for q, (c, x) in enumerate(zip(at, ijk))]
    return out


def step_us(s, n=8):
    best = 1e9
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.tstep = 1
        a.record()
        s.step(n)
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / n)
    return best


@pytest.mark.parametrize("shape,npml,each", [((64, 96, 96), 0, 60), ((20, 16, 32), 3, 33), ((64, 96, 96), 6, 15)])
def test_long_lists(shape, npml, each):
    src = spread(shape, each)
    a, b = (solver(shape, coefs(shape), sources=src, npml=npml, fused=f, max_steps=10) for f in (True, False))
    for s in (a, b):
        s.step(3)
    assert_same(a, b)
    one = solver(shape, coefs(shape), npml=npml, max_steps=10)
    one.step(1)
    assert step_us(a) < 3 * step_us(one)


@pytest.mark.parametrize("planes,fits", [(32, True), (36, False)])
def test_layouts_counted_in_chunks_of_48_planes(planes, fits):
    """Which layouts are refused does not follow the shorter x chunks of small grids:
    two rows of `planes` sources in the tile of rows 8 .. 23."""
    shape = (64, 64, 64)
    src = [("ez", (i, j, 20), lambda t: 1e-3 * t) for i in range(10, 10 + planes) for j in (10, 20)]
    s = solver(shape, coefs(shape), sources=src, npml=6, max_steps=4)
    if fits:
        s.step(1)
    else:
        with pytest.raises(ValueError, match="capacity"):
            s.step(1)
