"""4th-order stage pairs: grids small enough to be all shell (the edge kernels
alone), and the tiled pair kernel with its shell on grids of that size (an x
chunk given by the caller), on chained and on plain launches.  Equal bit for bit
to the one-launch-per-stage path; the tiled cases also run on the bounds-checked
build, in a child process (this file as a program)."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
pytestmark = pytest.mark.gpu

NAMES = ("ex", "ey", "ez", "hx", "hy", "hz")
# (shape, npml, faces, x_chunk)
TILED = [((40, 60, 132), 5, 0x3F, 40), ((26, 70, 164), 6, 0x30, 9), ((30, 80, 68), 3, 0x0C, 30),
         ((24, 100, 201), 4, 0x3F, 8), ((20, 44, 66), 0, 0x3F, 0)]
AUTO = [((12, 9, 7), 0, 0x3F, 0), ((30, 31, 44), (4, 6, 9), 0x3F, 0), ((22, 40, 67), 4, 0x21, 0),
        ((5, 4, 4), 0, 0x3F, 0), ((96, 128, 128), 0, 0x3F, 0), ((97, 128, 128), 0, 0x3F, 0),
        ((162, 161, 164), 6, 0x3F, 0), ((128, 128, 132), 6, 0x3F, 0), ((200, 210, 204), 6, 0x3F, 0)]


def check(shape, npml, faces, x_chunk):
    from fdtd_accelerate_gb300.symplectic import COURANT, SymplecticSolver
    rng = np.random.default_rng(9)
    ce = [(COURANT / 24 / rng.uniform(1.0, 4.0, shape)).astype(np.float32) for _ in range(3)]
    init = {k: (0.1 * rng.standard_normal(shape)).astype(np.float32) for k in NAMES}
    nx, ny, nz = shape
    src = [("ez", (nx // 2, ny // 2, nz // 2), lambda t: np.sin(0.3 * t)), ("ex", (3, 2, nz - 2), lambda t: 0.1 * t)]
    runs = []
    for fused in (True, False):
        s = SymplecticSolver(shape, ce=ce, npml=npml, faces=faces, sources=src, max_steps=5, fused=fused,
                             x_chunk=x_chunk)
        s.set_fields(**init)
        s.step(3)
        runs.append(s)
    torch.cuda.synchronize()
    a, b = runs
    a.check_status()
    for k in NAMES:
        assert torch.equal(a.fields[k], b.fields[k]), (shape, k)
    for q in range(6):
        if a.cpml.psi_e[q] is not None:
            assert torch.equal(a.cpml.psi_e[q], b.cpml.psi_e[q]) and torch.equal(a.cpml.psi_h[q], b.cpml.psi_h[q]), shape


@pytest.mark.parametrize("case", TILED + AUTO, ids=str)
def test_pairs_equal_stages(case):
    check(*case)


def test_tiled_pairs_on_the_checked_build():
    from fdtd_accelerate_gb300 import buildlib
    buildlib.build(check=True)
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], env=dict(os.environ, FDTD_GB300_CHECKED="1"),
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and r.stdout.split()[-1] == "0", r.stdout[-2000:] + r.stderr[-4000:]


if __name__ == "__main__":
    from fdtd_accelerate_gb300 import _native as N
    assert N.CHECKED
    for case in TILED:
        check(*case)
    torch.cuda.synchronize()
    word = C.c_uint64(0)
    N.call("fdtd_debug_check", C.byref(word))
    print(word.value)
