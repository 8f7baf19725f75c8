"""The persistent CG and BiCGStab (grid-wide and one cluster per instance) against the per-phase
kernels: the same bits, on the shapes where the work split can go wrong: rows of four, odd rows,
partial tiles, one cell thick blocks, rotated connections, instances of 1 to 33 tiles (a cluster
holds at most 32), batches of few and many systems, best iterates of solves cut off early."""
import pytest
import torch

import phipict_b200 as pb
from phipict_b200 import _C
from phipict_b200.solvers import BICGSTAB, CG, solver_for
from cases import duct_3d, hartmann_2d, periodic_box_3d, rotated_pair_2d, rotated_pair_3d, seeded_state

pytestmark = pytest.mark.gpu

CASES = {
    "row4_3d": lambda **k: duct_3d(16, 12, 8, 2, **k),
    "odd_3d": lambda **k: duct_3d(13, 11, 9, 3, **k),
    "thin_3d": lambda **k: duct_3d(20, 1, 24, 1, **k),
    "wide_3d": lambda **k: duct_3d(48, 40, 20, 2, **k),        # 76 tiles: the grid kernel
    "wide_odd_3d": lambda **k: duct_3d(37, 25, 23, 2, **k),
    "rotated_2d": lambda **k: rotated_pair_2d(16, **k),
    "rotated_3d": lambda **k: rotated_pair_3d(**k),
    "rotated_swapped_3d": lambda **k: rotated_pair_3d((8, 12, 8), 16, swapped=True, **k),  # rows of four beside it
    "rotated_wide_3d": lambda **k: rotated_pair_3d((32, 24, 28), 36, **k),                 # the grid kernel
    "periodic_3d": lambda **k: periodic_box_3d(32, 36, 40, **k),
    "one_tile": lambda **k: hartmann_2d(32, 24, **k),
    "two_tiles": lambda **k: hartmann_2d(64, 32, **k),
    "three_tiles_odd": lambda **k: hartmann_2d(51, 53, **k),
    "sixteen_tiles_odd": lambda **k: hartmann_2d(129, 121, **k),
    "seventeen_tiles": lambda **k: hartmann_2d(128, 129, **k),  # two tiles per CTA from here
    "thirty_two_tiles": lambda **k: hartmann_2d(181, 181, **k),
    "thirty_three_tiles": lambda **k: hartmann_2d(184, 180, **k),
    "batch_of_copies": lambda **k: hartmann_2d(33, 31, batch=3, **k),
}


def _assemble(dom, seed):
    ts = torch.tensor([0.01], dtype=torch.float64)
    _C.SetupAdvectionMatrix(dom, ts, 0)
    _C.SetupPressureMatrix(dom, ts)


def _rhs(dom, n, nrhs, seed):
    g = torch.Generator().manual_seed(seed)
    b = torch.randn(n * nrhs, generator=g, dtype=torch.float64).to(dom.getDtype()).to(dom.getDevice())
    dom._subtract_mean(b, nrhs)
    return b


def _solve(dom, kind, nrhs, A, b, tol, maxit, mode, best=False, ctas=0):
    s = solver_for(dom, kind, dom.getDtype(), nrhs, tag=f"m{mode}c{ctas}")
    x = torch.zeros_like(b)
    s.solve(A, b, x, tol, maxit, return_best=best, use_graph=mode, ctas_per_sm=ctas)
    return x, s.results()


def _same(a, b):
    return torch.equal(a[0], b[0]) and [(i.usedIterations, i.finalResidual, i.status) for i in a[1]] == [
        (i.usedIterations, i.finalResidual, i.status) for i in b[1]]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("case", list(CASES))
def test_persistent_solvers_match_per_phase_kernels(cuda, case, dtype):
    dom = CASES[case](dtype=dtype)
    seeded_state(dom, 5, scale=0.2)
    dom.PrepareSolve()
    _assemble(dom, 5)
    n = dom.numCells()
    d = dom.getSpatialDims()
    tol = 1e-4
    b = _rhs(dom, n, 1, 7)
    ref = _solve(dom, CG, 1, dom._P_st, b, tol, 3000, 1)
    assert all(i.converged for i in ref[1])
    assert _same(_solve(dom, CG, 1, dom._P_st, b, tol, 3000, 2), ref)          # a cluster per instance up to 32 tiles
    assert _same(_solve(dom, CG, 1, dom._P_st, b, tol, 3000, 2, ctas=1), ref)  # the grid kernel
    # cut off before convergence: the best iterate
    ref = _solve(dom, CG, 1, dom._P_st, b, 1e-30, 7, 1, best=True)
    for ctas in (0, 1):
        assert _same(_solve(dom, CG, 1, dom._P_st, b, 1e-30, 7, 2, best=True, ctas=ctas), ref)
    for nrhs in (1, d):
        b = _rhs(dom, n, nrhs, 9)
        ref = _solve(dom, BICGSTAB, nrhs, dom._C_st, b, 1e-5, 500, 1)
        assert all(i.converged for i in ref[1])
        assert _same(_solve(dom, BICGSTAB, nrhs, dom._C_st, b, 1e-5, 500, 2), ref)
        if nrhs > 1:
            ref = _solve(dom, CG, nrhs, dom._P_st, b, tol, 3000, 1)
            assert _same(_solve(dom, CG, nrhs, dom._P_st, b, tol, 3000, 2), ref)


@pytest.mark.parametrize("sizes", [((16, 12), (33, 20), (64, 48)),
                                   ((16, 12), (13, 9), (64, 48), (33, 20), (8, 8), (6, 10), (40, 36), (21, 7), (12, 12), (96, 50), (5, 4))],
                         ids=["few", "many"])
def test_persistent_solvers_of_a_batch(cuda, sizes):
    """Instances that stop after different counts, in one launch: the per-phase kernels' bits."""
    doms = []
    for k, (nx, ny) in enumerate(sizes):
        m = hartmann_2d(nx, ny)
        seeded_state(m, 60 + k, scale=0.2)
        m.PrepareSolve()
        doms.append(m)
    batch = pb.DomainBatch(doms)
    _assemble(batch, 3)
    b = _rhs(batch, batch.numCells(), 1, 3)
    ref = _solve(batch, CG, 1, batch._P_st, b, 1e-6, 3000, 1)
    assert len({i.usedIterations for i in ref[1]}) > 1
    for ctas in (0, 1):
        assert _same(_solve(batch, CG, 1, batch._P_st, b, 1e-6, 3000, 2, ctas=ctas), ref)
    b = _rhs(batch, batch.numCells(), 2, 4)
    ref = _solve(batch, BICGSTAB, 2, batch._C_st, b, 1e-8, 500, 1)
    assert _same(_solve(batch, BICGSTAB, 2, batch._C_st, b, 1e-8, 500, 2), ref)


@pytest.mark.parametrize("kind", [CG, BICGSTAB], ids=["cg", "bicgstab"])
def test_block_tables_that_do_not_fit_shared_memory(cuda, kind):
    """500 instances: the tables of their blocks go to global memory; still the per-phase kernels' bits."""
    dom = hartmann_2d(9, 7)
    dom.setBatchSize(500)
    dom.PrepareSolve()
    g = torch.Generator().manual_seed(2)
    v = dom.getBlocks()[0].velocity
    v.copy_((1.0 + 0.2 * torch.randn(v.shape, generator=g, dtype=torch.float64)).to(v.device, v.dtype))
    _assemble(dom, 2)
    nrhs = 1 if kind == CG else 2
    A, tol = (dom._P_st, 1e-6) if kind == CG else (dom._C_st, 1e-8)
    b = _rhs(dom, dom.numCells(), nrhs, 3)
    ref = _solve(dom, kind, nrhs, A, b, tol, 1000, 1)
    assert all(i.converged for i in ref[1])
    assert _same(_solve(dom, kind, nrhs, A, b, tol, 1000, 2, ctas=1), ref)


@pytest.mark.parametrize("kind,nrhs,instances", [(CG, 1, 1281), (CG, 2, 641), (BICGSTAB, 1, 1281), (BICGSTAB, 2, 641)])
def test_more_systems_than_a_cta_keeps_states_of_are_refused(cuda, kind, nrhs, instances):
    """160 KB of states, 1280 systems: the persistent mode refuses more whichever kernel would run."""
    dom = hartmann_2d(5, 4)
    dom.setBatchSize(instances)
    dom.PrepareSolve()
    b = torch.ones(dom.numCells() * nrhs, dtype=torch.float64, device=cuda)
    A = dom._P_st if kind == CG else dom._C_st
    with pytest.raises(RuntimeError, match="too many systems"):
        _solve(dom, kind, nrhs, A, b, 1e-6, 10, 2)


def test_a_batch_of_more_clusters_than_fit_at_a_time(cuda):
    """127 instances of one tile and one of 25: clusters are sized for 25 tiles, so that few are resident,
    and 19 waves of them take 2.4 times the grid kernel's time. The default must not be that slow (the
    bits are the same either way)."""
    doms = []
    for k in range(128):
        m = hartmann_2d(*((24 + k % 8, 20 + k % 11) if k < 127 else (160, 160)))
        seeded_state(m, k, scale=0.2)
        m.PrepareSolve()
        doms.append(m)
    batch = pb.DomainBatch(doms)
    _assemble(batch, 3)
    b = _rhs(batch, batch.numCells(), 1, 3)

    def run(ctas):
        s = solver_for(batch, CG, torch.float64, 1, tag=f"w{ctas}")
        best = float("inf")
        for _ in range(5):
            x = torch.zeros_like(b)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            s.solve(batch._P_st, b, x, 1e-200, 40, use_graph=2, ctas_per_sm=ctas)
            e1.record()
            e1.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return x, best

    (x0, t0), (x1, t1) = run(0), run(3)
    assert torch.equal(x0, x1)
    assert t0 < 1.5 * t1, (t0, t1)


# Tiles per worker group at one group per SM: more than 8 (the sums of a phase are flushed in its middle,
# forwards and backwards), more than 16 (the tile list goes on in global memory), and more than 256 tiles
# of one instance (several rounds of loads in its sums)
LONG = {
    "rows_of_four_2d": lambda **k: hartmann_2d(1600, 1600, **k),  # 2500 tiles
    "odd_2d": lambda **k: hartmann_2d(1601, 1597, **k),           # 2497 tiles
    "rows_of_four_3d": lambda **k: duct_3d(128, 104, 100, 1, **k),  # 1300 tiles
    "odd_3d": lambda **k: duct_3d(137, 139, 133, 1, **k),          # 2474 tiles
    "large_3d": lambda **k: duct_3d(256, 184, 180, 1, **k),        # 8280 tiles, past 2^23 cells
}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=["f32", "f64"])
@pytest.mark.parametrize("case", list(LONG))
def test_long_tile_lists_match_per_phase_kernels(cuda, case, dtype):
    dom = LONG[case](dtype=dtype)
    seeded_state(dom, 5, scale=0.2)
    dom.PrepareSolve()
    _assemble(dom, 5)
    assert dom.desc().ntiles > 8 * 148
    d = dom.getSpatialDims()
    for kind, A, nrhs, its in ((CG, dom._P_st, 1, 7), (BICGSTAB, dom._C_st, 1, 4), (BICGSTAB, dom._C_st, d, 4)):
        b = _rhs(dom, dom.numCells(), nrhs, 7)
        ref = _solve(dom, kind, nrhs, A, b, 1e-30, its, 1)
        assert all(i.isFiniteResidual for i in ref[1])
        for ctas in (0, 1):
            assert _same(_solve(dom, kind, nrhs, A, b, 1e-30, its, 2, ctas=ctas), ref), (kind, nrhs, ctas)
