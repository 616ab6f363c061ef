"""The face-flux kernels read 32-byte state rows with one load where the arrays start on a 32-byte boundary.
dndsg_eval_rhs_noalloc also takes a caller's arrays that start on a 16-byte one: those rows take two loads.
Meshes with more faces than the split kernel takes, so that k_face_flux itself runs."""
import numpy as np
import pytest

from dnds_b200 import geometry as G
from dnds_b200 import mesh as M
from dnds_b200 import settings as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset", ["vortex", "riemann"])
@pytest.mark.parametrize("precision", [0, 1])
def test_rows_on_16_byte_boundaries(preset, precision):
    import torch

    from dnds_b200.solver import BUF_U, BUF_UREC, Solver

    if preset == "vortex":
        m = M.vortex_mesh(78, True, jitter=0.2, seed=1234)  # 18,252 faces
        u0 = G.isentropic_vortex(m)
    else:
        m = M.riemann_mesh(78)
        u0 = G.quadrant_states(m, S.RIEMANN_2D_STATES)
    assert m.n_faces > 16384
    s = Solver(m, S.preset(preset), precision=precision)
    s.set_u(u0)
    s.ReconstructionJacobiStep(3)
    s.EvaluateDt(0.4)
    ref = s.EvaluateRHS(0.01)
    size = 8 if precision == 0 else 4
    rec = s.get_urec()
    for du, dr in [(0, 0), (16, 0), (0, 16), (16, 16)]:
        bu = torch.empty(32 * m.n_cells + 64, dtype=torch.uint8, device="cuda")
        br = torch.empty(20 * size * m.n_cells + 64, dtype=torch.uint8, device="cuda")
        out = torch.full((m.n_cells, 4), float("nan"), dtype=torch.float64, device="cuda")
        u = bu[du : du + 32 * m.n_cells].view(torch.float64)
        r = br[dr : dr + 20 * size * m.n_cells].view(torch.float64 if precision == 0 else torch.float32)
        assert u.data_ptr() % 32 == du and r.data_ptr() % 32 == dr
        u.copy_(torch.as_tensor(np.ascontiguousarray(s.get_u(), dtype=np.float64).reshape(-1)))
        r.copy_(torch.as_tensor(np.ascontiguousarray(rec, dtype=np.float64).reshape(-1)).to(r.dtype))
        s.EvaluateRHS_noalloc(u.data_ptr(), r.data_ptr(), out.data_ptr(), 0.01)
        torch.cuda.synchronize()
        # the same sums over the same rows: the tolerance of the allocation-free entry against the regular one
        assert np.abs(out.cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
    s.close()
