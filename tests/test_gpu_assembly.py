"""The central assembly kernels at the edges of their work split, against the oracle with the checks
and bars of test_gpu_parity: rows of four and odd rows, tiles cut short, a block of several
tiles, blocks one cell thick, 3D connections that turn and mirror the axes, more tiles than resident
CTAs (a CTA then takes several)."""
import pytest
import torch

import test_gpu_parity as parity
from cases import duct_3d, hartmann_2d, rotated_pair_3d, seeded_state
from phipict_b200 import _C

pytestmark = pytest.mark.gpu

SHAPES = {
    "rows_of_four_3d": lambda dt: duct_3d(8, 12, 16, 2, dtype=dt),
    "odd_tiles_3d": lambda dt: duct_3d(19, 17, 9, 3, dtype=dt),
    "one_thick_3d": lambda dt: duct_3d(1, 6, 5, 3, dtype=dt),
    "one_cell_tail_2d": lambda dt: hartmann_2d(41, 25, dtype=dt),   # 1025 cells
    "full_tile_2d": lambda dt: hartmann_2d(32, 32, dtype=dt),
    "rotated_3d": lambda dt: rotated_pair_3d(dtype=dt),
    "rotated_swapped_3d": lambda dt: rotated_pair_3d(swapped=True, dtype=dt),
}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_central_assembly_at_the_edges_of_its_tiles(cuda, monkeypatch, shape, dtype):
    monkeypatch.setitem(parity.CASES, shape, SHAPES[shape])
    parity.test_advection_and_pressure_assembly(cuda, shape, dtype)
    if dtype == torch.float64:
        parity.test_potential_assembly_and_current_density(cuda, shape, dtype)


@pytest.mark.parametrize("swapped", [False, True], ids=["turned", "swapped"])
def test_central_assembly_across_turned_connections_of_distorted_blocks(cuda, monkeypatch, swapped):
    """Metrics that differ on the two sides of the connection: the neighbour's component, sign and
    metric index all count."""
    monkeypatch.setitem(parity.CASES, "distorted", lambda dt: rotated_pair_3d(swapped=swapped, distorted=True, dtype=dt))
    parity.test_advection_and_pressure_assembly(cuda, "distorted", torch.float64)
    parity.test_potential_assembly_and_current_density(cuda, "distorted", torch.float64)


def _everything(dom, seed, batch):
    """Every central assembly output, per instance, of a domain whose instances are all alike."""
    import ctypes as ct

    from phipict_b200 import _lib

    n, d, dt = dom.getTotalSize(), dom.getSpatialDims(), dom.getDtype()
    g = torch.Generator().manual_seed(seed)
    field = torch.randn(d * n, generator=g, dtype=torch.float64).to(dt).cuda()
    p = torch.randn(n, generator=g, dtype=torch.float64).to(dt).cuda()
    dom._u_block.copy_((1 + 0.2 * field).reshape(1, d, n).expand(batch, d, n))
    ts = torch.tensor([0.01], dtype=torch.float64)
    _C.SetupAdvectionMatrix(dom, ts, 0)
    _C.SetupAdvectionVelocity(dom, ts, 0, False)
    dom.velocityResult.copy_(field.repeat(batch))
    _C.SetupPressureCorrection(dom, ts, 0, False, False)
    dom.pressureResult.copy_(p.repeat(batch))
    S = _lib.stream_ptr(dom.getDevice())
    corrected = torch.empty_like(dom.pressureRHS)
    _lib.call("phb_correct_velocity", ct.byref(dom.desc()), dom.pressureResult.data_ptr(), dom.pressureRHS.data_ptr(),
              dom.A.data_ptr(), corrected.data_ptr(), S)
    eb = torch.tensor([[0.3, 1.0, -0.5]] * batch, dtype=torch.float64, device="cuda")
    uxb, rhs = torch.empty(batch * 3 * n, dtype=dt, device="cuda"), torch.empty(batch * n, dtype=dt, device="cuda")
    _lib.call("phb_uxb_epot_rhs", ct.byref(dom.desc()), dom._u_block.data_ptr(), eb.data_ptr(), uxb.data_ptr(), rhs.data_ptr(), S)
    epot = torch.empty(batch * n, dtype=dt, device="cuda")
    _lib.call("phb_epot_rhs", ct.byref(dom.desc()), dom.velocityResult.data_ptr(), epot.data_ptr(), S)
    out = {"C": dom._C_st.view(-1, batch, n).transpose(0, 1), "P": dom._P_st.view(-1, batch, n).transpose(0, 1)}
    for k, v in dict(A=dom.A, rhs=dom.velocityRHS, hbya=dom.pressureRHS, div=dom.pressureRHSdiv, corrected=corrected, uxb=uxb,
                     uxb_rhs=rhs, epot=epot).items():
        out[k] = v.view(batch, -1)
    return out


# Tiles (all instances) at which the kernels with 2, 3 or 4 resident CTAs per SM take: quarter tiles in runs of up
# to six, quarter tiles one grid apart (3D), whole tiles
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32], ids=["f64", "f32"])
@pytest.mark.parametrize("shape,per", [("duct", 10), ("rotated", 19), ("channel", 9)])
@pytest.mark.parametrize("tiles", [400, 1000, 1172])
def test_every_share_of_the_tiles_gives_the_same_bits(cuda, shape, per, tiles, dtype):
    """A batch of equal instances against a single one, whose few tiles are taken in quarters."""
    make = {"duct": lambda: duct_3d(27, 19, 18, 1, dtype=dtype), "rotated": lambda: rotated_pair_3d((20, 24, 16), 28, dtype=dtype),
            "channel": lambda: hartmann_2d(97, 85, dtype=dtype)}[shape]
    outs = []
    for batch in (1, tiles // per):
        dom = make()
        if batch > 1:
            dom.setBatchSize(batch)
        dom.PrepareSolve()
        assert dom.desc().ntiles == per * batch
        outs.append(_everything(dom, 7, batch))
    for k, many in outs[1].items():
        assert torch.isfinite(many).all(), k
        assert torch.equal(outs[0][k].expand_as(many), many), k


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
