"""4th-order stage pairs on tiny grids, whose edge kernels take a thread for each
component: equal to the stage kernels bit for bit, on both sides of the size where
that ends, with sources and merged passes of two H stages."""
import pytest
import torch

from tests.test_gpu_symp_layout import assert_same, coefs, solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,npml", [((4, 4, 4), 0), ((5, 7, 8), 0), ((20, 18, 16), (4, 3, 6)), ((58, 22, 36), 6),
                                        ((48, 64, 64), 8), ((49, 64, 64), 8), ((20, 40, 45), (6, 0, 0))])
def test_tiny_grids(shape, npml):
    src = [(c, tuple(min(n - 1, n // 2 + q) for n in shape), lambda t, q=q: 1e-3 * (q + 1) * t)
           for q, c in enumerate(("ex", "ey", "ez", "ex"))]
    a, b = (solver(shape, coefs(shape), npml=npml, sources=src, fused=f, max_steps=160) for f in (True, False))
    for s in (a, b):
        s.step(3)
        s.step(130)
    assert_same(a, b)
    for q in range(6):
        if b.cpml.psi_e[q] is not None:
            assert torch.equal(a.cpml.psi_e[q], b.cpml.psi_e[q]) and torch.equal(a.cpml.psi_h[q], b.cpml.psi_h[q])
