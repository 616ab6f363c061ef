"""The scan-order LU-SGS walk with U5 in clusters of blocks and in wide batches (levels of more than one batch of 32
cells; the meshes of the other SA tests have narrower ones) against the oracle's sequential sweep
(DNDS_FV_EulerEvaluator.cpp:1149-1357).  C-meshes of ni x nj cells: in the natural order the mean level has
ni nj / (ni + nj - 1) cells, and a part is walked by a cluster of one block per 8 of them."""
import numpy as np
import pytest

from dnds_b200 import mesh as M
from dnds_b200 import settings as S


@pytest.mark.gpu
@pytest.mark.parametrize("na,nw,nj,order,parts", [
    (96, 52, 160, "natural", 1),  # 200 x 160, 89 cells a level: 16 blocks
    (40, 30, 80, "natural", 1),   # 100 x 80, 45: 8 blocks
    (96, 52, 160, "natural", 2),  # two parts of 100 x 160, 62: 8 blocks each, ghosts in the backward sweep
    (96, 52, 160, "line", 1),     # 161 levels of 199, four neighbours at the wake cut: runs of cells
    (64, 32, 40, "random", 1),    # random cell numbers: one block, wide batches
])
def test_walk_with_u5_matches_sequential_sweep(oracle_lib, na, nw, nj, order, parts):
    """Pseudo-time iterations: 1e-9 of the state, as in the other comparisons of RANS-SA iterations (the source runs
    through exp and log)."""
    from dnds_b200.solver import Solver

    m = M.naca0012_cmesh(na, nw, nj, first=1e-3, far=10.0)
    scan = M.line_scan_order(m) if order == "line" else None
    if order == "random":
        m, _ = M.renumber(m, np.random.default_rng(5).permutation(m.n_cells))
    cfg = S.naca0012_sa(0.15, 10.0, 1e5)
    u0 = np.tile(np.array(cfg["eulerSetting"]["farFieldStaticValue"]), (m.n_cells, 1))
    part = (np.arange(m.n_cells) * parts) // m.n_cells
    s = Solver(m, cfg, precision=0)
    s.lusgs_set_order(1, scan)
    o = oracle_lib.Oracle(m, cfg, n_threads=4)
    if parts > 1:
        s.lusgs_set_parts(part, parts)
        o.set_lusgs_parts(part)
    s.set_u(u0)
    s.bdf_begin()
    o.set_u(u0)
    for _ in range(6):
        res, _ = s.implicit_iteration(20.0)
        inc = o.implicit_iteration(20.0, u0, scan2cell=scan)
        assert abs(res[4] - np.abs(inc[:, 4]).sum()) < 1e-8 * max(res[4], 1e-300)
    ref = o.get_u()
    assert np.abs(s.get_u() - ref).max() < 1e-9 * np.abs(ref).max()
    assert s.status()[0] == 0
    s.close()
