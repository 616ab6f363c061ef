"""Steps captured through a caller's stream (include/dndsg.h allows it): the caller's graph holds plain launches,
as the library's own step graphs do (a programmatic edge in a graph of small passes costs more than it saves),
and replays the steps of plain calls."""
import numpy as np
import pytest

from dnds_b200 import geometry as G
from dnds_b200 import mesh as M
from dnds_b200 import settings as S


def _solver(flow, n, precision, stream):
    from dnds_b200.solver import Solver

    if flow == "vortex":
        m, cfg = M.vortex_mesh(n, True, jitter=0.2), S.preset("vortex")
        u0 = G.isentropic_vortex(m)
    else:
        m, cfg = M.riemann_mesh(n), S.preset("riemann")
        u0 = G.quadrant_states(m, S.RIEMANN_2D_STATES)
    s = Solver(m, cfg, precision=precision, stream=stream)
    s.set_u(u0)
    return s


# 24: a thread per Gauss point; 96: a thread per face, still programmatic launches outside a capture
@pytest.mark.gpu
@pytest.mark.parametrize("flow,n,precision", [("vortex", 24, 0), ("vortex", 96, 1), ("riemann", 32, 1)])
def test_captured_step(flow, n, precision):
    import torch
    from cuda.bindings import runtime as rt

    stream = torch.cuda.Stream().cuda_stream
    s, ref = _solver(flow, n, precision, stream), _solver(flow, n, precision, None)
    for _ in range(3):
        s.ssprk3_step(0.5)
    torch.cuda.synchronize()
    ok = rt.cudaError_t.cudaSuccess
    assert rt.cudaStreamBeginCapture(stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0] == ok
    for _ in range(2):  # an even number of buffer swaps
        s.ssprk3_step(0.5)
    err, graph = rt.cudaStreamEndCapture(stream)
    assert err == ok
    count = rt.cudaGraphGetEdges_v2(graph)[-1]
    err, _, _, data, _ = rt.cudaGraphGetEdges_v2(graph, count)
    assert err == ok and count >= 2 * 10 - 1
    assert not any(int(d.type) == int(rt.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic) for d in data)
    err, run = rt.cudaGraphInstantiate(graph, 0)
    assert err == ok
    for _ in range(3):
        assert rt.cudaGraphLaunch(run, stream)[0] == ok
    torch.cuda.synchronize()
    for _ in range(3 + 6):
        ref.ssprk3_step(0.5)
    assert np.array_equal(s.get_u(), ref.get_u()) and s.time == ref.time
    rt.cudaGraphExecDestroy(run)
    rt.cudaGraphDestroy(graph)
    s.close()
    ref.close()
