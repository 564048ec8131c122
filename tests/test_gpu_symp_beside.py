"""4th-order stage pairs on grids whose shell H kernel runs beside the pair kernel:
equal to the stage kernels bit for bit, on a stream of the caller's, in a CUDA graph,
and when the plan goes while its last pass may still run."""
import pytest
import torch

from tests.test_gpu_symp_layout import assert_same, coefs, solver

pytestmark = pytest.mark.gpu

# (shape, npml, x_chunk): the range's ends for aligned rows, and an x chunk given on a small grid
CASES = [((150, 168, 168), 6, 0), ((200, 204, 204), 4, 0), ((162, 161, 164), (0, 0, 8), 0), ((40, 60, 132), 5, 40)]


@pytest.mark.parametrize("shape,npml,x_chunk", CASES)
def test_on_a_stream_and_in_a_graph(shape, npml, x_chunk):
    a, g, b = (solver(shape, coefs(shape), npml=npml, x_chunk=x_chunk, fused=f, max_steps=16) for f in (True, True, False))
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        for n in (1, 5):
            a.step(n)
        held = {k: v.clone() for k, v in a.fields.items()}
        a.close()
    g.step(1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        g.step(5)
    graph.replay()
    b.step(6)
    torch.cuda.synchronize()
    a.check_status()
    for k in held:
        assert torch.equal(held[k], b.fields[k]), k
    assert_same(a, b)
    assert_same(g, b)
    for q in range(6):
        if b.cpml.psi_e[q] is not None:
            for s in (a, g):
                assert torch.equal(s.cpml.psi_e[q], b.cpml.psi_e[q]) and torch.equal(s.cpml.psi_h[q], b.cpml.psi_h[q])
