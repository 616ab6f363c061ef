"""The schedules of the scan-order LU-SGS walk (dnds_b200/csrc/dndsg_lusgs_sched.hpp) on the host:
tests/lusgs_walk_check.cpp builds them for grids of quads and triangles, walks them with the blocks of a part
in random turns, and checks that every increment a cell reads (ring, mailbox or global memory) is that of the
neighbour the reference's sequential sweep reads (DNDS_FV_EulerEvaluator.cpp:1149-1357), that no value is
overwritten before its last reader and that the blocks never wait in a circle.  On the GPU: wide levels,
several blocks per part and three used neighbours against the sequential oracle."""
import os
import subprocess

import numpy as np
import pytest

from dnds_b200 import geometry as G
from dnds_b200 import mesh as M
from dnds_b200 import settings as S

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = tmp_path_factory.mktemp("walk") / "lusgs_walk_check"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "dnds_b200", "csrc"),
                        os.path.join(ROOT, "tests", "lusgs_walk_check.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(exe)


# nx, ny, triangles, parts, order (0 natural, 1 reversed, 2 shuffled cells and parts, 3 shuffled cells, 4 even lines then odd
# ones), blocks per part (-1: one, wide batches; < -1: of consecutive cells)
@pytest.mark.parametrize("case", [(1, 1, 0, 1, 0, 1), (5, 3, 0, 4, 1, 8), (33, 31, 0, 1, 0, 2), (30, 20, 1, 3, 2, 4), (70, 64, 0, 1, 1, 16),
                                  (64, 70, 1, 2, 0, 8), (100, 90, 1, 1, 2, 16), (256, 64, 0, 16, 0, 1), (512, 128, 0, 1, 0, 16),
                                  (1, 1, 0, 1, 0, -1), (500, 300, 0, 1, 0, -1), (65, 63, 0, 2, 1, -1), (120, 100, 0, 1, 2, -1), (100, 70, 1, 3, 2, -1),
                                  (100, 90, 0, 1, 3, -16), (60, 64, 1, 1, 3, -8), (64, 100, 0, 1, 4, -16), (64, 96, 0, 2, 4, -4)])
def test_schedule(check, case):
    for seed in (1, 2):
        r = subprocess.run([check, *map(str, case), str(seed)], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout
        assert "ok 2" in r.stdout


@pytest.mark.parametrize("case,want", [
    ((512, 128, 0, 1, 0), "16x32 16x32"),   # levels of 103 cells
    ((512, 1200, 0, 1, 0), "16x32 16x32"),  # 2,400 mailbox slots: with U5 they fit beside records of three neighbours
    ((512, 2048, 0, 1, 0), "1x64 1x64"),    # 4,096 fit beside neither
    ((256, 64, 0, 16, 0), "1x32 1x32"),     # levels of one batch
    ((128, 128, 0, 1, 2), "16x32 16x32"),   # shuffled: by runs of the scan order nearly every cell goes to every block
    ((512, 128, 0, 1, 4), "16x32 16x32"),   # lines, even ones first
    ((128, 900, 0, 1, 4), "1x64 1x64"),     # the same, a cluster's blocks would wait on one another at every level
    ((4800, 64, 0, 75, 0), "1x64 1x64"),    # as many parts as half the multiprocessors, levels of up to 64 cells
])
def test_blocks_per_part_and_batch_width(check, case, want):
    r = subprocess.run([check, *map(str, case), "0", "1"], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.split() == want.split(), r.stdout


# clusters of blocks with runs of cells (a shuffled order), and wide batches (shuffled cells, where neither runs of
# the order nor of cells fit, every neighbour out of the ring; and 75 parts with levels of up to 64 cells)
@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny,tri,parts,shuffle", [(96, 90, False, 1, "order"), (60, 50, True, 2, "order"), (128, 64, False, 1, "cells"),
                                                     (70, 65, True, 1, "cells"), (64, 4800, False, 75, None)])
def test_cell_runs_and_wide_batches_match_sequential_sweep(oracle_lib, nx, ny, tri, parts, shuffle):
    """Two pseudo-time iterations, as above."""
    from dnds_b200.solver import Solver

    m = M.structured_grid(nx, ny, 10.0, 10.0 * ny / nx, triangles=tri, jitter=0.15, periodic=False, bc=M.BC_FARFIELD)
    rng = np.random.default_rng(nx)
    if shuffle == "cells":
        m, _ = M.renumber(m, rng.permutation(m.n_cells))
    cfg = S.preset("vortex", eulerSetting={"farFieldStaticValue": [1.0, 1.0, 1.0, 3.5]})
    u0 = np.tile([1.0, 1.0, 1.0, 3.5], (m.n_cells, 1)) * (1 + 0.02 * rng.uniform(size=(m.n_cells, 4)))
    scan = rng.permutation(m.n_cells) if shuffle == "order" else None
    part = (np.arange(m.n_cells) * parts) // m.n_cells
    s = Solver(m, cfg, precision=0)
    s.lusgs_set_order(1, scan)
    if parts > 1:
        s.lusgs_set_parts(part, parts)
    s.set_u(u0)
    s.bdf_begin()
    o = oracle_lib.Oracle(m, cfg, n_threads=4)
    o.set_u(u0)
    if parts > 1:
        o.set_lusgs_parts(part)
    for _ in range(2):
        s.implicit_iteration(20.0)
        o.implicit_iteration(20.0, u0, scan2cell=scan)
    assert np.abs(s.get_u() - o.get_u()).max() < 1e-12 * np.abs(o.get_u()).max()
    assert s.status()[0] == 0
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cells,nx,ny,parts", [("quad", 96, 90, 1), ("tri", 60, 50, 1), ("tri", 64, 33, 3), ("quad", 7, 5, 1)])
def test_walk_matches_sequential_sweep(oracle_lib, cells, nx, ny, parts):
    """One forward and backward sweep through pseudo-time iterations: FP64 against the oracle's sequential
    order, 1e-12 of the state (sums of at most four terms per level, in another order)."""
    from dnds_b200.solver import Solver

    m = M.structured_grid(nx, ny, 10.0, 10.0, triangles=cells == "tri", jitter=0.15, periodic=False, bc=M.BC_FARFIELD)
    cfg = S.preset("vortex", eulerSetting={"farFieldStaticValue": [1.0, 1.0, 1.0, 3.5]})
    u0 = G.isentropic_vortex(m)
    part = (np.arange(m.n_cells) * parts) // m.n_cells
    s = Solver(m, cfg, precision=0)
    s.lusgs_set_order(1)
    s.lusgs_set_parts(part, parts)
    s.set_u(u0)
    s.bdf_begin()
    o = oracle_lib.Oracle(m, cfg, n_threads=4)
    o.set_u(u0)
    if parts > 1:
        o.set_lusgs_parts(part)
    for _ in range(2):
        s.implicit_iteration(20.0)
        o.implicit_iteration(20.0, u0)
    assert np.abs(s.get_u() - o.get_u()).max() < 1e-12 * np.abs(o.get_u()).max()
    s.close()
