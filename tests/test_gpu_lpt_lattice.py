"""Particles written at their lattice points (pmb_lpt_lattice) against
pmb_lpt on the generated grid: the same sums per particle, so bit for bit.
Grids whose rows are not whole groups of four, thin grids, orders 0 to 2."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 8, 8), (7, 6, 5), (4, 9, 10), (2, 3, 2), (5, 4, 67), (16, 2, 128)])
@pytest.mark.parametrize("order", [0, 1, 2])
@pytest.mark.parametrize("mesh", [1, 2])
def test_lattice_particles_bitwise(shape, order, mesh):
    import pmpp_b200 as pb
    from pmpp_b200 import lpt as pl
    from pmpp_b200._lib import call, lib
    from pmpp_b200.runtime import stream_handle
    conf = pb.Configuration(4.0, shape, mesh, a_start=0.1, lpt_order=order, device="cuda")
    cos = pb.boltzmann(pb.SimpleLCDM(conf))
    g = torch.Generator(device="cuda").manual_seed(1)
    gx, gy, gz = shape
    modes = torch.fft.rfftn(torch.randn(shape, generator=g, device="cuda")).contiguous()
    res = pl.lpt_full(modes, cos, conf)
    ref = pb.Particles.gen_grid(conf, vel=True)
    fac, _ = cos.lpt_factors(conf.a_start)
    fields = torch.empty((6, ) + shape, device="cuda")
    index = torch.empty(conf.ptcl_num, dtype=torch.int64, device="cuda")
    ws = torch.empty(lib().pmb_lpt_workspace_bytes(gx, gy, gz), dtype=torch.uint8, device="cuda")
    tab = conf.spectral_tables("particle", modes.device)
    call("pmb_lpt", modes.data_ptr(), gx, gy, gz, float(conf.ptcl_spacing), float(conf.ptcl_cell_vol), tab.data_ptr(),
         order, float(fac[0, 0]), float(fac[0, 2]), float(fac[1, 0]), float(fac[1, 2]), ref.pmid.data_ptr(),
         ref.disp.data_ptr(), ref.vel.data_ptr(), conf.ptcl_num, float(conf.cell_size), fields.data_ptr(),
         index.data_ptr(), ws.data_ptr(), ws.numel(), stream_handle(modes.device))
    for name in ("pmid", "disp", "vel"):
        assert torch.equal(getattr(res.ptcl, name), getattr(ref, name)), name
    assert torch.equal(res.index, index)
    for m in range(3 * order):  # the fields of the orders in use
        assert torch.equal(res.fields[m], fields[m]), m


def _conf():
    import pmpp_b200 as pb
    return pb.Configuration(4.0, (7, 6, 5), 2, a_start=0.1, device="cuda")


def _same(tables, conf):
    from pmpp_b200 import Particles
    pm, dp = Particles.lattice_axes(conf, torch.device("cuda"))
    return torch.equal(tables[0], torch.cat(pm)) and torch.equal(tables[1], torch.cat(dp))


def test_axis_tables_are_complete_when_kept():
    """Another stream may read the kept tables at once, so the work that makes them has ended."""
    conf = _conf()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        tables = conf.lattice_tables("cuda")
        assert side.query()
    assert conf.lattice_tables("cuda")[0] is tables[0]
    assert _same(tables, conf)


def test_axis_tables_of_a_capture_are_its_own():
    conf = _conf()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        held = conf.lattice_tables("cuda")
    assert held[0] is not conf.lattice_tables("cuda")[0]  # nothing that only a replay fills is kept
    assert _same(conf.lattice_tables("cuda"), conf)
    graph.replay()
    assert _same(held, conf)
