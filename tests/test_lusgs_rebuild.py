"""Rebuilding the scan-order LU-SGS schedule: an error leaves the schedule in force as it was."""
import numpy as np
import pytest

from dnds_b200 import mesh as M
from dnds_b200 import settings as S


def _setup():
    m = M.structured_grid(512, 256, 20.0, 10.0, triangles=False, jitter=0.1, periodic=False, bc=M.BC_FARFIELD)
    cfg = S.preset("vortex", eulerSetting={"farFieldStaticValue": [1.0, 1.0, 1.0, 3.5]})
    u0 = np.tile([1.0, 1.0, 1.0, 3.5], (m.n_cells, 1)) * (1 + 0.02 * np.random.default_rng(1).uniform(size=(m.n_cells, 4)))
    return m, cfg, u0


def _fill_device(rt):
    """Takes the free device memory, down to pieces of 64 KB."""
    held, size = [], 1 << 36
    while size >= 1 << 16:
        err, p = rt.cudaMalloc(size)
        if err == rt.cudaError_t.cudaSuccess:
            held.append(p)
        else:
            size //= 2
    return held


@pytest.mark.gpu
@pytest.mark.parametrize("change", ["order", "parts"])
def test_a_rebuild_that_finds_no_memory(oracle_lib, change):
    from cuda.bindings import runtime as rt

    from dnds_b200.solver import DndsgError, Solver

    m, cfg, u0 = _setup()
    s = Solver(m, cfg, precision=0)
    s.lusgs_set_order(1)
    s.set_u(u0)
    s.bdf_begin()
    o = oracle_lib.Oracle(m, cfg, n_threads=4)
    o.set_u(u0)
    s.implicit_iteration(20.0)
    o.implicit_iteration(20.0, u0)
    reverse, part = np.arange(m.n_cells)[::-1].copy(), (np.arange(m.n_cells) * 4) // m.n_cells
    held = _fill_device(rt)
    try:
        with pytest.raises(DndsgError, match="out of memory"):
            if change == "order":
                s.lusgs_set_order(1, reverse)
            else:
                s.lusgs_set_parts(part, 4)
    finally:
        for p in held:
            rt.cudaFree(p)
    s.implicit_iteration(20.0)  # in the order from before
    o.implicit_iteration(20.0, u0)
    assert np.abs(s.get_u() - o.get_u()).max() < 1e-12 * np.abs(o.get_u()).max()
    # a part with too many levels is refused; the order and the parts in force stay too
    s.lusgs_set_parts(part, 4)
    o.set_lusgs_parts(part)
    s.implicit_iteration(20.0)
    o.implicit_iteration(20.0, u0)
    assert np.abs(s.get_u() - o.get_u()).max() < 1e-12 * np.abs(o.get_u()).max()
    snake = np.arange(m.n_cells).reshape(256, 512)
    snake[1::2] = snake[1::2, ::-1]
    with pytest.raises(DndsgError, match="levels per part"):
        s.lusgs_set_order(1, snake.ravel())
    assert s.lusgs_set_parts(part, 4) == 2 * (512 + 64 - 1)  # still the natural order
    s.implicit_iteration(20.0)
    o.implicit_iteration(20.0, u0)
    assert np.abs(s.get_u() - o.get_u()).max() < 1e-12 * np.abs(o.get_u()).max()
    s.close()
