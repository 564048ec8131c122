"""Reverse step with 4 cells a thread (rows on 16-byte boundaries) against the
one-cell kernels (taken for bases off them): ragged row ends, slabs that begin
and end inside a group, both z slabs in one group, gradient boxes that cut
groups, psi rows on and off the boundaries, repeated monitor points.  Equal bit
for bit."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,npml,faces,box", [
    ((14, 13, 16), 4, 0x3F, None), ((14, 12, 13), 4, 0x3F, (2, 1, 3, 9, 10, 6)), ((12, 14, 10), 4, 0x3F, None),
    ((9, 8, 131), (2, 3, 7), 0x3F, (0, 0, 5, 9, 8, 2)), ((12, 10, 12), (0, 4, 5), 0x2D, None),
    ((6, 5, 7), 0, 0x3F, None), ((5, 6, 3), 0, 0x3F, None), ((14, 13, 20), 5, 0x12, (3, 3, 0, 4, 4, 20)),
])
def test_reverse_step_groups(shape, npml, faces, box):
    from fdtd_accelerate_gb300 import _native as N
    from fdtd_accelerate_gb300.cpml import CpmlLayer
    nx, ny, nz = shape
    pitch = (nz + 3) // 4 * 4
    layer = CpmlLayer(shape, npml, faces)
    gen = torch.Generator(device="cuda").manual_seed(4)

    def rnd(n):
        return torch.randn(n, generator=gen, device="cuda")

    size = nx * ny * pitch
    fields = {k: rnd(n * size) for k, n in (("lf", 6), ("ce", 3), ("gce", 3), ("hp", 3))}
    psis = {k: [rnd(t.numel()) if t is not None else None for t in layer.psi_e[0]] for k in ("lpe", "lph", "pe", "we", "wh")}
    mons = torch.tensor([[1, 2, 1], [1, 2, 1], [nx - 1, 0, nz - 1], [1, 2, 1], [nx, 0, 0]], dtype=torch.int32, device="cuda")
    comp = torch.tensor([2, 2, 4, 1, 0], dtype=torch.int32, device="cuda")
    vals = rnd(5)
    results = []
    for off in (0, 1):  # bases on, then off the 16-byte boundaries
        f = {k: torch.empty(v.numel() + 1, device="cuda")[off:off + v.numel()] for k, v in fields.items()}
        for k in f:
            f[k].copy_(fields[k])
        ps = {k: [t.clone() if t is not None else None for t in v] for k, v in psis.items()}
        st = N.AdjointState()
        for q in range(6):
            st.lf[q] = f["lf"][q * size:].data_ptr()
            for arr, k in ((st.lpsi_e, "lpe"), (st.lpsi_h, "lph"), (st.w_e, "we"), (st.w_h, "wh")):
                arr[q] = ps[k][q].data_ptr() if ps[k][q] is not None else None
        for q in range(3):
            st.grad_ce[q] = f["gce"][q * size:].data_ptr()
        g = N.Grid(nx, ny, nz, ny * pitch, pitch)
        cp = layer.struct()
        pts = N.Points()
        pts.n, pts.ijk, pts.comp = 5, mons.data_ptr(), comp.data_ptr()
        hp = (C.c_void_p * 3)(*[f["hp"][q * size:].data_ptr() for q in range(3)])
        ce = (C.c_void_p * 3)(*[f["ce"][q * size:].data_ptr() for q in range(3)])
        pe = (C.c_void_p * 6)(*[t.data_ptr() if t is not None else None for t in ps["pe"]])
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        for _ in range(2):
            args = [C.byref(g), C.byref(cp), C.byref(st), hp, pe, ce, C.byref(pts), C.c_void_p(vals.data_ptr())]
            if box is None:
                N.call("fdtd_adjoint_step_f32", *args, stream)
            else:
                N.call("fdtd_adjoint_step_region_f32", *args, (C.c_int64 * 6)(*box), stream)
        torch.cuda.synchronize()
        results.append((f, ps))
    (fa, pa), (fb, pb) = results
    for k in ("lf", "gce"):
        assert torch.equal(fa[k], fb[k]), k     # the padding of the rows among it
    for k in ("lpe", "lph"):
        for a, b in zip(pa[k], pb[k]):
            assert a is None or torch.equal(a, b), k
    assert np.isfinite(fa["lf"].cpu().numpy()).all()
