"""The persistent multigrid-preconditioned CG (one cooperative kernel) against the same solver as
per-phase kernels (host loop), over the grids where its work split can go wrong: rows of four and
two cells and odd rows, blocks one cell thick, single-cell aggregates, connected blocks with rotated
axes, grids of several tiles per block, quarter and whole tiles on the finest level, item lists longer
than shared memory keeps, more instances than warps in a block, block tables in global memory, and
solves cut off before convergence (best iterate)."""
import pytest
import torch

import phipict_b200 as pb
from phipict_b200 import _C
from phipict_b200.amg import AmgHierarchy
from phipict_b200.solvers import CG, solver_for
from cases import duct_3d, hartmann_2d, periodic_box_3d, rotated_pair_2d, rotated_pair_3d, seeded_state

pytestmark = pytest.mark.gpu

CASES = {
    "row4_3d": lambda: duct_3d(16, 12, 8, 2, dtype=torch.float32),
    "row2_3d": lambda: duct_3d(14, 10, 6, 2, dtype=torch.float32),
    "odd_3d": lambda: duct_3d(13, 11, 9, 3, dtype=torch.float32),
    "row4_odd_3d": lambda: duct_3d(12, 11, 9, 2, dtype=torch.float32),
    "thin_z": lambda: duct_3d(24, 20, 1, 2, dtype=torch.float32),
    "thin_y": lambda: duct_3d(20, 1, 24, 1, dtype=torch.float32),
    "row4_2d": lambda: hartmann_2d(32, 24, dtype=torch.float32),
    "odd_2d": lambda: hartmann_2d(33, 31, dtype=torch.float32),
    "rotated_2d": lambda: rotated_pair_2d(16, dtype=torch.float32),
    "rotated_3d": lambda: rotated_pair_3d(dtype=torch.float32),
    "rotated_swapped_3d": lambda: rotated_pair_3d((8, 12, 8), 16, swapped=True, dtype=torch.float32),
    # rows of four on the finest restriction (131,072 cells and more), quarter tiles elsewhere
    "wide_3d": lambda: duct_3d(64, 48, 24, 2, dtype=torch.float32),
    "wide_2d": lambda: hartmann_2d(512, 384, dtype=torch.float32),
    "tiles_odd_3d": lambda: duct_3d(37, 25, 23, 2, dtype=torch.float32),
    # at least 296 tiles: whole tiles on the finest level, rows of four ...
    "whole_tiles_3d": lambda: duct_3d(32, 72, 70, 2, dtype=torch.float32),
    "whole_tiles_periodic_3d": lambda: periodic_box_3d(64, 72, 70, dtype=torch.float32),
    "whole_tiles_2d": lambda: hartmann_2d(640, 512, dtype=torch.float32),
    # ... and cell by cell: odd rows, and rows of four whose block meets a turned connection
    "whole_tiles_odd_3d": lambda: duct_3d(67, 71, 65, 1, dtype=torch.float32),
    "whole_tiles_odd_2d": lambda: hartmann_2d(641, 487, dtype=torch.float32),
    "whole_tiles_rotated_3d": lambda: rotated_pair_3d((64, 80, 32), 56, dtype=torch.float32),
}


def _system(dom, seed):
    seeded_state(dom, seed, scale=0.2)
    dom.PrepareSolve()
    ts = torch.tensor([0.01], dtype=torch.float64)
    _C.SetupAdvectionMatrix(dom, ts, 0)
    _C.SetupPressureMatrix(dom, ts)
    n = dom.getTotalSize()
    b = torch.randn(n, generator=torch.Generator().manual_seed(seed + 1), dtype=torch.float64)
    return (b - b.mean()).to(torch.float32).to(dom.getDevice())


def _solve(dom, A, b, tol, maxit, mode, h, best=False, ctas=0):
    s = solver_for(dom, CG, torch.float32, 1, tag=f"pcg{mode}{ctas}")
    x = torch.zeros_like(b)
    s.solve(A, b, x, tol, maxit, return_best=best, use_graph=mode, amg=h, ctas_per_sm=ctas)
    return x, s.results()


@pytest.mark.parametrize("case", list(CASES))
def test_persistent_pcg_matches_per_phase_kernels(cuda, case):
    dom = CASES[case]()
    b = _system(dom, 11)
    h = AmgHierarchy(dom)
    h.setup(dom._P_st)
    tol = 1e-4 * float(b.norm() / b.numel() ** 0.5)
    x0, i0 = _solve(dom, dom._P_st, b, tol, 500, 0, h)
    x2, i2 = _solve(dom, dom._P_st, b, tol, 500, 2, h)
    assert i0[0].converged and i2[0].converged
    assert abs(i0[0].usedIterations - i2[0].usedIterations) <= 1
    # both stop at the same float32 residual; the iterates differ by that residual through the inverse
    assert float((x2 - x0).double().norm() / x0.double().norm()) < 1e-3
    # a fixed iteration count: the same iterate up to float32 rounding of a few sweeps
    x0, _ = _solve(dom, dom._P_st, b, 0.0, 4, 0, h, best=True)
    x2, r2 = _solve(dom, dom._P_st, b, 0.0, 4, 2, h, best=True)
    assert not r2[0].converged and r2[0].isFiniteResidual
    assert float((x2 - x0).double().norm() / x0.double().norm()) < 1e-4
    # the result does not depend on the grid
    x1, _ = _solve(dom, dom._P_st, b, 0.0, 4, 2, h, best=True, ctas=1)
    assert torch.equal(x1, x2)


def test_persistent_pcg_of_a_batch(cuda):
    """Twelve instances of mixed alignment and size that stop after different counts."""
    doms = []
    for k, (nx, ny) in enumerate([(16, 12), (13, 9), (64, 48), (33, 20), (8, 8), (6, 10), (40, 36), (21, 7), (12, 12), (96, 50), (5, 4), (28, 16)]):
        d = hartmann_2d(nx, ny, dtype=torch.float32)
        seeded_state(d, 60 + k, scale=0.2)
        d.PrepareSolve()
        doms.append(d)
    batch = pb.DomainBatch(doms)
    ts = torch.tensor([0.01], dtype=torch.float64)
    _C.SetupAdvectionMatrix(batch, ts, 0)
    _C.SetupPressureMatrix(batch, ts)
    g = torch.Generator().manual_seed(3)
    b = torch.randn(batch.numCells(), generator=g).cuda()
    batch._subtract_mean(b, 1)
    h = AmgHierarchy(batch)
    h.setup(batch._P_st)
    x0, i0 = _solve(batch, batch._P_st, b, 1e-4, 500, 0, h)
    x2, i2 = _solve(batch, batch._P_st, b, 1e-4, 500, 2, h)
    assert all(i.converged for i in i0) and all(i.converged for i in i2)
    assert len({i.usedIterations for i in i2}) > 1
    for e in range(len(doms)):
        sl = batch.instance_slice(e)
        assert abs(i0[e].usedIterations - i2[e].usedIterations) <= 1, e
        assert float((x2[sl] - x0[sl]).double().norm() / x0[sl].double().norm()) < 2e-3, e


# more than eight items per worker group at one group per SM (148 x 8 tiles): the lists go on in global
# memory, are visited backwards every other pass, and the sums of a pass are flushed in its middle
LONG = {
    "rows_of_four_3d": lambda: duct_3d(128, 104, 100, 1, dtype=torch.float32),  # 1300 tiles
    "odd_3d": lambda: duct_3d(111, 107, 109, 1, dtype=torch.float32),           # 1265 tiles
    "rows_of_four_2d": lambda: hartmann_2d(1600, 1600, dtype=torch.float32),    # 2500 tiles
    "odd_2d": lambda: hartmann_2d(1109, 1201, dtype=torch.float32),             # 1301 tiles
}


@pytest.mark.parametrize("case", list(LONG))
def test_persistent_pcg_with_long_item_lists(cuda, case):
    dom = LONG[case]()
    b = _system(dom, 12)
    assert dom.desc().ntiles > 8 * 148
    h = AmgHierarchy(dom)
    h.setup(dom._P_st)
    # a fixed iteration count: the same iterate up to float32 rounding of a few sweeps
    x0, _ = _solve(dom, dom._P_st, b, 0.0, 5, 0, h, best=True)
    x1, r1 = _solve(dom, dom._P_st, b, 0.0, 5, 2, h, best=True, ctas=1)
    assert not r1[0].converged and r1[0].isFiniteResidual
    assert float((x1 - x0).double().norm() / x0.double().norm()) < 1e-4
    for ctas in (0, 2):
        x2, _ = _solve(dom, dom._P_st, b, 0.0, 5, 2, h, best=True, ctas=ctas)
        assert torch.equal(x1, x2)


@pytest.mark.parametrize("size", [(20, 12), (13, 9)], ids=["rows_of_four", "odd"])
def test_persistent_pcg_with_block_tables_in_global_memory(cuda, size):
    """300 instances: the tables of all levels exceed the 48 KB that shared memory keeps."""
    dom = hartmann_2d(*size, dtype=torch.float32)
    dom.setBatchSize(300)
    dom.PrepareSolve()
    g = torch.Generator().manual_seed(2)
    v = dom.getBlocks()[0].velocity
    v.copy_((1.0 + 0.2 * torch.randn(v.shape, generator=g)).to(v.device))
    ts = torch.tensor([0.01], dtype=torch.float64)
    _C.SetupAdvectionMatrix(dom, ts, 0)
    _C.SetupPressureMatrix(dom, ts)
    b = torch.randn(dom.numCells(), generator=g).cuda()
    dom._subtract_mean(b, 1)
    h = AmgHierarchy(dom)
    h.setup(dom._P_st)
    assert h.nlevels * dom.desc().nblocks * 128 > 48 * 1024
    x0, i0 = _solve(dom, dom._P_st, b, 1e-4, 500, 0, h)
    x2, i2 = _solve(dom, dom._P_st, b, 1e-4, 500, 2, h)
    assert all(i.converged for i in i0) and all(i.converged for i in i2)
    n = dom.getTotalSize()
    for e in range(300):
        assert abs(i0[e].usedIterations - i2[e].usedIterations) <= 1, e
        sl = slice(e * n, (e + 1) * n)
        assert float((x2[sl] - x0[sl]).double().norm() / x0[sl].double().norm()) < 2e-3, e
