"""What a caller of SymplecticSolver holds on rows that are no multiple of 4
floats is what it holds on aligned ones."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

NAMES = ("ex", "ey", "ez", "hx", "hy", "hz")


def solver(shape, ce, sources=None, max_steps=300, **kw):
    from fdtd_accelerate_gb300.symplectic import SymplecticSolver
    rng = np.random.default_rng(3)
    s = SymplecticSolver(shape, ce=ce, max_steps=max_steps,
                         sources=sources or [("ez", tuple(n // 2 for n in shape), lambda t: 1e-3 * t)], **kw)
    s.set_fields(**{k: (0.1 * rng.standard_normal(shape)).astype(np.float32) for k in NAMES})
    return s


def coefs(shape, seed=4):
    rng = np.random.default_rng(seed)
    return [torch.from_numpy((0.743 / 24 / rng.uniform(1.0, 4.0, shape)).astype(np.float32)).cuda() for _ in range(3)]


def assert_same(a, b):
    torch.cuda.synchronize()
    for k in NAMES:
        assert torch.equal(a.fields[k], b.fields[k]), k


@pytest.mark.parametrize("how", ["step", "step_stages", "step_unfused"])
@pytest.mark.parametrize("nz", [44, 45])
def test_edited_coefficients_reach_the_next_call(nz, how):
    shape = (20, 40, nz)
    ce = coefs(shape)
    s = solver(shape, ce, ch=[0.75 * c for c in coefs(shape, 5)] if how != "step" else None)
    getattr(s, how)(128)
    for c in ce:
        c.mul_(0.5)
    before = {k: v.clone() for k, v in s.fields.items()}
    getattr(s, how)(128)
    r = solver(shape, [c.clone() for c in ce], ch=s.ch)
    r.set_fields(**before)
    r.tstep = 129
    getattr(r, how)(128)
    assert_same(s, r)


@pytest.mark.parametrize("nz", [44, 45])
def test_fields_are_dense(nz):
    """The fields of any grid are contiguous arrays, which the per-call functions
    take together with arrays of the caller's."""
    from fdtd_accelerate_gb300 import symplectic as S
    shape = (20, 40, nz)
    ce = coefs(shape)
    s = solver(shape, ce)
    held = s.fields
    s.step(128)
    for k in NAMES:
        assert s.fields[k].is_contiguous() and s.fields[k].data_ptr() == held[k].data_ptr()
        s.fields[k].view(-1)[0] += 1.0
    e = [torch.zeros(shape, device="cuda") for _ in range(3)]
    h = s.f[3:]
    S.update_e(*shape, S.DL[0], *e, *h, *ce)
    r = [torch.zeros(shape, device="cuda") for _ in range(3)]
    S.update_e(*shape, S.DL[0], *r, *[x.clone() for x in h], *ce)
    torch.cuda.synchronize()
    for a, b in zip(e, r):
        assert torch.equal(a, b)


def test_many_sources_in_one_tile():
    """More sources than the pair kernel stages for a tile: the stage kernels take
    any number of them."""
    shape = (20, 40, 45)
    src = [(c, (i, j, 6), lambda t, q=q: 1e-3 * q * t)
           for q, (c, i, j) in enumerate((c, i, j) for c in ("ex", "ez") for i in range(2, 18) for j in (3, 5, 7))]
    a, b = (solver(shape, coefs(shape), sources=src, fused=fused) for fused in (True, False))
    for s in (a, b):
        s.step(128)
    assert_same(a, b)


@pytest.mark.parametrize("first", [True, False])
def test_step_under_capture(first):
    """step() of odd rows in a CUDA graph, as the solver's first call (the stage
    kernels) and after one that made the pair plan."""
    shape = (20, 40, 45)
    a, b = (solver(shape, coefs(shape)) for _ in range(2))
    for s in (a, b):
        if not first:
            s.step(128)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        a.step(128)
    assert a._plan_ready() != first
    graph.replay()
    b.step(128)
    assert_same(a, b)


def test_no_memory_for_the_copies():
    """A grid whose state fits the device and whose second state does not."""
    shape = (64, 80, 81)
    a, b = (solver(shape, coefs(shape), npml=(4, 0, 0), fused=fused) for fused in (True, False))
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (8 << 20)) / total)
    try:
        a.step(128)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    b.step(128)
    assert_same(a, b)
    for q in range(2):
        assert torch.equal(a.cpml.psi_e[q], b.cpml.psi_e[q]) and torch.equal(a.cpml.psi_h[q], b.cpml.psi_h[q])


@pytest.mark.parametrize("shape,npml,n,pairs", [
    ((20, 40, 45), 0, 1, False), ((20, 40, 45), 0, 127, False), ((20, 40, 45), 0, 128, True),
    ((90, 90, 91), 0, 128, False), ((64, 100, 121), 3, 128, False), ((160, 160, 165), 0, 15, False),
    ((160, 160, 165), 0, 16, True), ((160, 160, 165), 6, 16, False), ((200, 204, 207), 6, 16, True),
    ((256, 256, 257), 6, 4, False), ((256, 256, 257), 6, 5, True)])
def test_short_runs_keep_the_stage_kernels(shape, npml, n, pairs):
    """Runs too short, or grids too small, to make up for the copies of the state
    neither make a plan nor allocate a second state."""
    a, b = (solver(shape, coefs(shape), npml=npml, fused=fused) for fused in (True, False))
    assert a.pair_path()
    for s in (a, b):
        s.step(n)
    assert a._plan_ready() == pairs and (a._pitched is not None) == pairs
    assert_same(a, b)


def test_two_h_stages_of_unlike_layers_are_refused():
    """A pass of two H stages whose layers differ: an error code, and the state as it was."""
    import ctypes as C
    from fdtd_accelerate_gb300 import _native as N
    from fdtd_accelerate_gb300.symplectic import CL, DL
    s = solver((20, 40, 44), coefs((20, 40, 44)), npml=4)
    s.step(1)
    before = {k: v.clone() for k, v in s.fields.items()}
    a, e, none, thin, half = s.cpml._structs[CL[0]], s.cpml._structs[DL[0]], N.Cpml(), N.Cpml(), N.Cpml()
    for other, npml, faces in ((thin, 3, 0x3F), (half, 4, 0x2F)):
        C.memmove(C.byref(other), C.byref(a), C.sizeof(a))
        other.npml[2], other.faces = npml, faces
    ref = lambda c: C.byref(c) if c is not None else None
    for ha, hb in ((a, None), (None, a), (a, none), (a, thin), (thin, a), (a, half)):
        st = N.lib().fdtd_symp_pair_run(s._pair, ref(ha), ref(hb), ref(e), CL[4], CL[0], 1, DL[0], float(s.ch), -1, None)
        assert st == N.FDTD_ERR_ARG
    assert N.lib().fdtd_symp_pair_plan_current(s._pair) == s._cur
    torch.cuda.synchronize()
    for k in NAMES:
        assert torch.equal(s.fields[k], before[k]), k


def test_pairs_and_stages_by_turns():
    """Long and short calls of one solver on odd rows, with an x layer (psi of both
    paths) and edits of the fields between the calls."""
    shape, npml = (20, 40, 45), (5, 0, 0)
    a, b = (solver(shape, coefs(shape), npml=npml, fused=fused, max_steps=400) for fused in (True, False))
    for n in (3, 128, 1, 129, 2):
        for s in (a, b):
            s.step(n)
            s.fields["ey"].mul_(0.5)
    assert a._plan_ready()
    assert_same(a, b)
    for q in range(2):
        assert torch.equal(a.cpml.psi_e[q], b.cpml.psi_e[q]) and torch.equal(a.cpml.psi_h[q], b.cpml.psi_h[q])
    a.check_status()
