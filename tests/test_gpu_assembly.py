"""The central assembly kernels at the edges of their work split, against the oracle with the checks
and bars of test_gpu_parity: rows of four and odd rows, tiles cut short, a block of several
tiles, blocks one cell thick, more tiles than resident CTAs (a CTA then takes several)."""
import pytest
import torch

import test_gpu_parity as parity
from cases import duct_3d, hartmann_2d, seeded_state
from phipict_b200 import _C

pytestmark = pytest.mark.gpu

SHAPES = {
    "rows_of_four_3d": lambda dt: duct_3d(8, 12, 16, 2, dtype=dt),
    "odd_tiles_3d": lambda dt: duct_3d(19, 17, 9, 3, dtype=dt),
    "one_thick_3d": lambda dt: duct_3d(1, 6, 5, 3, dtype=dt),
    "one_cell_tail_2d": lambda dt: hartmann_2d(41, 25, dtype=dt),   # 1025 cells
    "full_tile_2d": lambda dt: hartmann_2d(32, 32, dtype=dt),
}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_central_assembly_at_the_edges_of_its_tiles(cuda, monkeypatch, shape, dtype):
    monkeypatch.setitem(parity.CASES, shape, SHAPES[shape])
    parity.test_advection_and_pressure_assembly(cuda, shape, dtype)
    if dtype == torch.float64:
        parity.test_potential_assembly_and_current_density(cuda, shape, dtype)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
def test_several_tiles_per_cta_give_the_values_of_one(cuda, dtype):
    """A batch of 1600 equal instances (more tiles than resident CTAs) has the matrix diagonal and
    right-hand side of a single one in every instance, bit for bit."""
    outs = []
    for batch in (1, 1600):
        dom = hartmann_2d(33, 5, dtype=dtype)
        if batch > 1:
            dom.setBatchSize(batch)
        dom.PrepareSolve()
        ref = hartmann_2d(33, 5, device="cpu", dtype=dtype)
        seeded_state(ref, 4)
        u = ref.getBlocks()[0].velocity[0].to(cuda)
        for b in range(batch):
            dom.getBlocks()[0].velocity[b].copy_(u)
        ts = torch.tensor([0.01], dtype=torch.float64)
        _C.SetupAdvectionMatrix(dom, ts, 0)
        _C.SetupAdvectionVelocity(dom, ts, 0, False)
        outs.append((dom.A.reshape(batch, -1).clone(), dom.velocityRHS.reshape(batch, -1).clone()))
    for one, many in zip(*outs):
        assert torch.equal(one.expand_as(many), many)
