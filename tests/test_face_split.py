"""Face passes on both sides of the face count from which one thread takes a whole face (below it a thread
takes one Gauss point, interior and boundary faces share a launch) and of programmatic launches: the residual,
local dt and two SSP-RK3 steps against the oracle.  90 x 90 quads have 16,380 faces, 91 x 90 have 16,561.
Tolerances as in tests/test_gpu_parity.py: FP64 1e-11 (one evaluation), FP32 bulk 2e-5 of the largest entry."""
import numpy as np
import pytest

from dnds_b200 import geometry as G
from dnds_b200 import mesh as M
from dnds_b200 import settings as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [1, 90, 91])
@pytest.mark.parametrize("riemann,bc", [("Roe", M.BC_WALL_EULER), ("HLLC", M.BC_FARFIELD)])
@pytest.mark.parametrize("precision", [0, 1])
def test_residual_and_steps(oracle_lib, nx, riemann, bc, precision):
    from dnds_b200.solver import Solver

    m = M.structured_grid(nx, 90, 10.0, 10.0, jitter=0.15, periodic=False, bc=bc)
    cfg = S.preset("vortex", eulerSetting={"riemannSolverType": riemann, "farFieldStaticValue": [1.0, 1.0, 1.0, 3.5]})
    u0 = G.isentropic_vortex(m)
    s = Solver(m, cfg, precision=precision)
    o = oracle_lib.Oracle(m, cfg, n_threads=4)
    s.set_u(u0)
    o.set_u(u0)
    s.ReconstructionJacobiStep(3)
    o.vr_step(3)
    s.EvaluateDt(0.5, use_local_dt=True)
    dt, dmin = o.eval_dt(0.5, use_local_dt=True)
    assert np.abs(s.get_dt() - dt).max() < 1e-13 * dt.max()
    rhs, ref = s.EvaluateRHS(0.0), o.eval_rhs(0.0)[0]
    assert np.abs(rhs - ref).max() < (2e-5 if precision else 1e-11) * np.abs(ref).max()
    for _ in range(2):
        _, dmin = o.eval_dt(0.5)
        s.ssprk3_step(0.5)
        o.ssprk3_step(dmin, 0.0)
    assert np.abs(s.get_u() - o.get_u()).max() < (1e-6 if precision else 1e-12) * np.abs(o.get_u()).max()
    assert s.status()[0] == 0
    s.close()
