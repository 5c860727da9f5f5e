"""Row sort at the edges of its launches: particle counts around the block's
1024, row counts around the grouping of unordered particles (1024 rows) and the
one-block scan (16384 rows), empty rows, long runs of one row, a drift; records, permutation and row offsets against the oracle's
binning (whole numbers, so exact)."""
import numpy as np
import pytest
import torch

from oracle import pm as opm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [(8, 8, 8), (16, 16, 3), (257, 1, 4), (32, 32, 2), (25, 41, 3), (128, 128, 4), (129, 128, 4), (1, 1, 8),
                                  (2, 3, 5), (300, 70, 2)])
@pytest.mark.parametrize("n", [1, 1023, 1025, 5000])
@pytest.mark.parametrize("drift", [None, 0.5])
def test_rows_records_and_offsets(mesh, n, drift):
    import pmpp_b200 as pb
    from pmpp_b200.cic import SortedParticles
    co = opm.Conf(2.0, mesh, mesh_shape=1)
    conf = pb.Configuration(2.0, mesh, 1, device="cuda")
    rng = np.random.default_rng(n)
    pmid = rng.integers(0, mesh, size=(n, 3)).astype(np.int16)
    pmid[n // 2:, :2] = pmid[0, :2]  # a long run of one row (and, displaced, of its neighbours)
    disp = rng.normal(0, 3.0, size=(n, 3)).astype(np.float32)
    vel = rng.normal(size=(n, 3)).astype(np.float32)
    d = torch.from_numpy(disp).cuda()
    kw = {} if drift is None else dict(drift_vel=torch.from_numpy(vel).cuda(), drift=drift)
    sp = SortedParticles(torch.from_numpy(pmid).cuda(), d, conf, **kw)
    if drift is not None:
        disp = disp + vel * np.float32(drift)
    assert np.array_equal(d.cpu().numpy(), disp)
    ref = opm.cell_key(pmid, disp, co)
    rec = sp.buf[:16 * n].view(torch.int32).reshape(n, 4).cpu().numpy()
    at = (16 * n + 255) // 256 * 256
    perm = sp.buf[at:at + 4 * n].view(torch.int32).cpu().numpy().astype(np.int64)
    at += (4 * n + 255) // 256 * 256
    rows = mesh[0] * mesh[1]
    offs = sp.buf[at:at + 4 * (rows + 1)].view(torch.int32).cpu().numpy()
    key = rec[:, 3].view(np.uint32).astype(np.int64)
    assert np.array_equal(np.sort(perm), np.arange(n))
    assert np.array_equal(key, ref[perm])
    assert np.array_equal(offs, np.searchsorted(np.sort(ref // mesh[2]), np.arange(rows + 1)))
    assert np.all(np.diff(key // mesh[2]) >= 0)
    q = disp / np.float32(co.cell_size)
    assert np.array_equal(rec[:, :3].view(np.float32), (q - np.floor(q))[perm])
