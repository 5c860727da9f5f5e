"""Deposit at the edges of its tiles and row strides: row lengths on and beside
the instantiated strides, meshes with remainders of the tile's rows, meshes of few
rows (one row per block once they are crowded) and of many, the
smallest meshes (a particle reaching one cell twice), values of every scale, an
output that is not 16-byte aligned, and one cell holding so many particles that
the 64-bit sums are taken.  The arithmetic is restated exactly
(helpers.fixed_point_scatter), so the comparison is bit for bit."""
import numpy as np
import pytest
import torch

from oracle import pm as opm
from tests.helpers import fixed_point_scatter

pytestmark = pytest.mark.gpu

MESHES = [(1, 1, 1), (2, 1, 3), (1, 2, 64), (3, 5, 65), (5, 2, 127), (9, 6, 128), (4, 7, 129), (6, 5, 192),
          (5, 5, 250), (7, 9, 256), (3, 6, 384), (5, 3, 512), (3, 3, 600), (2, 5, 768), (5, 2, 1024), (2, 2, 1500),
          (1, 3, 4096)]
# rows enough that 40000 particles are not a crowd
WIDE = [(37, 43, 3), (40, 37, 64), (37, 42, 65), (38, 40, 128), (41, 39, 192), (37, 41, 250), (39, 38, 256),
        (38, 39, 384), (41, 50, 512)]


def _particles(mesh, n, seed, crowd):
    import pmpp_b200 as pb
    co = opm.Conf(2.0, mesh, mesh_shape=1)
    conf = pb.Configuration(2.0, mesh, 1, device="cuda")
    rng = np.random.default_rng(seed)
    pmid = rng.integers(0, mesh, size=(n, 3)).astype(np.int16)
    disp = rng.normal(0, 4.0, size=(n, 3)).astype(np.float32)
    disp[:n // 50] = 0.0  # on the cell faces
    if crowd:
        pmid[n // 8:], disp[n // 8:] = pmid[0], disp[0]
    return co, conf, pmid, disp, rng


def _check(got, ref):
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("mesh", MESHES + WIDE)
@pytest.mark.parametrize("n,crowd", [(300, False), (40000, False), (40000, True)])
def test_density_bit_exact(mesh, n, crowd):
    from pmpp_b200.cic import SortedParticles
    co, conf, pmid, disp, _ = _particles(mesh, n, 1, crowd)
    sp = SortedParticles(torch.from_numpy(pmid).cuda(), torch.from_numpy(disp).cuda(), conf)
    for val in (8.0, -0.7):
        ref = fixed_point_scatter(pmid, disp, co, np.full(n, val, np.float32))
        _check(sp.scatter(val_const=val)[0].cpu().numpy(), ref)


@pytest.mark.parametrize("mesh", MESHES + WIDE)
@pytest.mark.parametrize("channels,scale", [(1, 1.0), (2, 1e-28), (3, 1.0), (3, 1e27), (4, 1e-5)])
def test_values_bit_exact_and_misaligned_output(mesh, channels, scale):
    from pmpp_b200.cic import SortedParticles
    n = 20000
    co, conf, pmid, disp, rng = _particles(mesh, n, 2, False)
    val = (rng.normal(size=(n, channels)) * 10.0**rng.integers(-3, 1, (n, 1)) * scale).astype(np.float32)
    sp = SortedParticles(torch.from_numpy(pmid).cuda(), torch.from_numpy(disp).cuda(), conf)
    ref = fixed_point_scatter(pmid, disp, co, val)
    v = torch.from_numpy(val).cuda()
    _check(sp.scatter(val=v, channels=channels).cpu().numpy(), ref)
    cells = channels * int(np.prod(mesh))
    out = torch.empty(cells + 4, device="cuda")[1:1 + cells].view((channels, ) + mesh)
    _check(sp.scatter(val=v, channels=channels, out=out).cpu().numpy(), ref)
