"""update_e / update_h with 4 cells a thread (rows on 16-byte boundaries) and
with one (others): contiguous and padded arrays, ragged row ends, single planes
and rows, ch arrays; the padding of a row is left alone.  Equal bit for bit to
the float32 NumPy expressions."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _numpy_e(f, c):
    ex, ey, ez, hx, hy, hz = f
    ex[:, :-1, :-1] += c[0][:, :-1, :-1] * (hz[:, 1:, :-1] - hz[:, :-1, :-1] - hy[:, :-1, 1:] + hy[:, :-1, :-1])
    ey[:-1, :, :-1] += c[1][:-1, :, :-1] * (hx[:-1, :, 1:] - hx[:-1, :, :-1] - hz[1:, :, :-1] + hz[:-1, :, :-1])
    ez[:-1, :-1, :] += c[2][:-1, :-1, :] * (hy[1:, :-1, :] - hy[:-1, :-1, :] - hx[:-1, 1:, :] + hx[:-1, :-1, :])


def _numpy_h(f, c):
    ex, ey, ez, hx, hy, hz = f
    hx[:, 1:, 1:] -= c[0][:, 1:, 1:] * (ez[:, 1:, 1:] - ez[:, :-1, 1:] - ey[:, 1:, 1:] + ey[:, 1:, :-1])
    hy[1:, :, 1:] -= c[1][1:, :, 1:] * (ex[1:, :, 1:] - ex[1:, :, :-1] - ez[1:, :, 1:] + ez[:-1, :, 1:])
    hz[1:, 1:, :] -= c[2][1:, 1:, :] * (ey[1:, 1:, :] - ey[:-1, 1:, :] - ex[1:, 1:, :] + ex[1:, :-1, :])


@pytest.mark.parametrize("shape,pitch,first", [
    ((9, 7, 8), 8, 0), ((5, 6, 4), 4, 0), ((3, 4, 129), 132, 0), ((4, 3, 130), 136, 0), ((2, 2, 131), 132, 0),
    ((6, 5, 3), 4, 0), ((1, 5, 16), 16, 0), ((5, 1, 16), 16, 0), ((4, 4, 1), 4, 0),
    ((4, 5, 13), 13, 0),    # unaligned rows
    ((4, 5, 12), 16, 1),    # aligned strides, unaligned base
])
@pytest.mark.parametrize("ch", [False, True])
def test_update_calls(shape, pitch, first, ch):
    from fdtd_accelerate_gb300 import api
    rng = np.random.default_rng(7)
    nx, ny, nz = shape
    host = [rng.standard_normal(shape).astype(np.float32) for _ in range(12)]
    dev, store = [], []
    for a in host:
        t = torch.full((nx * ny * pitch + 8,), 7.0, device="cuda")
        v = t[first:first + nx * ny * pitch].view(nx, ny, pitch)[:, :, :nz]
        v.copy_(torch.from_numpy(a))
        store.append((t, t.clone()))
        dev.append(v)
    f, ce, chs = host[:6], host[6:9], host[9:] if ch else [np.float32(0.5) * np.ones(shape, np.float32)] * 3
    for _ in range(2):
        api.update_e(*dev[:6], *dev[6:9])
        api.update_h(*dev[:6], *(dev[9:] if ch else ()))
        _numpy_e(f, ce)
        _numpy_h(f, chs)
    for n, (v, a) in enumerate(zip(dev, host)):
        np.testing.assert_array_equal(v.cpu().numpy(), a, err_msg=str(n))
    for (t, before), v in zip(store, dev):
        v.fill_(0)
        w = before[first:first + nx * ny * pitch].view(nx, ny, pitch)[:, :, :nz]
        w.fill_(0)
        assert torch.equal(t, before)  # nothing outside the array was written


@pytest.mark.parametrize("shape,npml,faces", [
    ((20, 18, 16), 4, 0x3F), ((12, 14, 132), (3, 5, 7), 0x3F),  # 4 cells a thread on the x and y slabs
    ((20, 18, 16), 4, 0x16), ((14, 12, 4), (4, 3, 0), 0x3F),    # some faces; rows of one group
    ((12, 13, 18), 4, 0x3F),                                     # psi rows off the 16-byte boundaries
])
@pytest.mark.parametrize("ch", [False, True])
def test_cpml_calls(shape, npml, faces, ch):
    """CpmlLayer.update_e / update_h with 4 cells a thread equal the one-cell
    kernels (taken for bases off the 16-byte boundaries), bit for bit; the
    one-cell kernels are compared with the oracle elsewhere."""
    from fdtd_accelerate_gb300.cpml import CpmlLayer
    rng = np.random.default_rng(9)
    layer = CpmlLayer(shape, npml, faces, device="cuda")
    nz4 = (shape[2] + 3) // 4 * 4
    f = []
    for _ in range(12):
        t = torch.zeros(shape[:2] + (nz4,), device="cuda")[:, :, :shape[2]]
        t.copy_(torch.from_numpy(rng.standard_normal(shape).astype(np.float32)))
        f.append(t)
    single = CpmlLayer(shape, npml, faces, device="cuda")
    off = []
    for t in f:
        b = torch.empty(t.numel() + 1, device="cuda")[1:].view(shape)
        b.copy_(t)
        off.append(b)
    for _ in range(3):
        layer.update_e(*f[:9])
        layer.update_h(*f[:6], *(f[9:] if ch else ()))
        single.update_e(*off[:9])
        single.update_h(*off[:6], *(off[9:] if ch else ()))
    for a, b in zip(f, off):
        assert torch.equal(a, b)
    for q in range(6):
        if layer.psi_h[q] is not None:
            assert torch.equal(layer.psi_e[0][q], single.psi_e[0][q]) and torch.equal(layer.psi_h[q], single.psi_h[q])
