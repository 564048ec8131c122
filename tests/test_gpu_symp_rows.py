"""4th-order stage pairs on rows that are no multiple of 4 floats (padded to a
16-byte pitch): equal the one-launch-per-stage path and the reference-shaped
calls bit for bit, with CPML faces, sources in the last cells of a row and ch
arrays (which keep the stage kernels); the padding stays zero."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

NAMES = ("ex", "ey", "ez", "hx", "hy", "hz")


@pytest.mark.parametrize("shape,npml,faces", [
    ((20, 100, 201), 4, 0x3F), ((40, 50, 66), 4, 0x15), ((20, 44, 67), 0, 0x3F), ((9, 8, 5), 0, 0x3F),
    ((26, 30, 34), 5, 0x3F),   # mostly shell: stage kernels
    ((30, 64, 97), 4, 0x30),
])
@pytest.mark.parametrize("ch_arrays", [False, True])
def test_padded_rows(shape, npml, faces, ch_arrays):
    from fdtd_accelerate_gb300.symplectic import COURANT, SymplecticSolver
    rng = np.random.default_rng(5)
    ce = [(COURANT / 24 / rng.uniform(1.0, 4.0, shape)).astype(np.float32) for _ in range(3)]
    ch = [(COURANT / 24 * rng.uniform(0.8, 1.0, shape)).astype(np.float32) for _ in range(3)] if ch_arrays else None
    init = {k: (0.1 * rng.standard_normal(shape)).astype(np.float32) for k in NAMES}
    nx, ny, nz = shape
    src = [("ez", (nx // 2, ny // 2, nz // 2), lambda t: np.sin(0.3 * t)), ("ex", (3, ny - 4, nz - 2), lambda t: 0.1 * t)]
    runs = []
    for how in ("pair", "stages", "calls"):
        s = SymplecticSolver(shape, ce=ce, ch=ch, npml=npml, faces=faces, sources=src, max_steps=6,
                             fused=how == "pair")
        assert s.pair_path() == (how == "pair" and not ch_arrays and shape != (26, 30, 34))
        s.set_fields(**init)
        (s.step_unfused if how == "calls" else s.step)(3)
        runs.append(s)
    torch.cuda.synchronize()
    a = runs[0]
    a.check_status()
    for b in runs[1:]:
        for k in NAMES:
            assert torch.equal(a.fields[k], b.fields[k]), k
        for q in range(6):
            if a.cpml.psi_e[q] is not None:
                assert torch.equal(a.cpml.psi_e[q], b.cpml.psi_e[q]) and torch.equal(a.cpml.psi_h[q], b.cpml.psi_h[q])
    for s in runs:
        for buf in s._buf:
            if buf is not None:
                whole = buf.as_strided((6, nx, ny, buf.stride(2)), buf.stride())
                assert not whole[..., nz:].any()
