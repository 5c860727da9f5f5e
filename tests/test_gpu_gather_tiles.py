"""Gather and position terms at the edges of their warps' 64-particle and the
blocks' 512-particle shares: counts beside both, masked slots, every optional
argument, against the oracle's float64 sums (2e-6 of the largest value: float32
weights and eight-term float32 sums) and, for the parts that must be the same
arithmetic, bit for bit."""
import numpy as np
import pytest
import torch

from oracle import pm as opm
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu

COUNTS = [1, 31, 63, 64, 65, 511, 512, 513, 1025, 3000]


def _sorted(n, masked, seed=0):
    import pmpp_b200 as pb
    from pmpp_b200.cic import SortedParticles
    mesh = (6, 5, 34)
    co = opm.Conf(2.0, mesh, mesh_shape=1)
    conf = pb.Configuration(2.0, mesh, 1, device="cuda")
    rng = np.random.default_rng(seed)
    pmid = rng.integers(0, mesh, size=(n, 3)).astype(np.int16)
    disp = rng.normal(0, 3.0, size=(n, 3)).astype(np.float32)
    valid = (rng.random(n) < 0.8) if masked else None
    v = None if valid is None else torch.from_numpy(valid.astype(np.uint8)).cuda()
    sp = SortedParticles(torch.from_numpy(pmid).cuda(), torch.from_numpy(disp).cuda(), conf, valid=v)
    return co, rng, pmid, disp, valid, sp, mesh


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("masked", [False, True])
def test_gather_and_kicks(n, channels, masked):
    from pmpp_b200._lib import call
    from pmpp_b200.runtime import stream_handle
    co, rng, pmid, disp, valid, sp, mesh = _sorted(n, masked)
    field = rng.normal(size=(channels, ) + mesh).astype(np.float32)
    f = torch.from_numpy(field).cuda()
    got = sp.gather(f)
    ref = opm.gather(pmid, disp, co, field, valid=valid)
    assert np.abs(got.cpu().numpy() - ref).max() < 2e-6 * np.abs(field).max()
    if masked:
        assert not got[torch.from_numpy(~valid).cuda()].abs().sum()
    if channels != 3:
        return
    v0 = torch.from_numpy(rng.normal(size=(n, 3)).astype(np.float32)).cuda()
    for k1, k2, keep in ((0.5, 0.0, True), (0.5, 0.25, True), (0.5, 0.25, False)):
        v, out = v0.clone(), torch.full_like(v0, 9.0)
        call("pmb_gather_rows2", sp.buf.data_ptr(), n, *mesh, 3, f.data_ptr(), out.data_ptr() if keep else None,
             v.data_ptr(), k1, k2, stream_handle(v.device))
        assert torch.equal(out, got) if keep else bool((out == 9).all())
        # two roundings per kick
        assert rel_err(v.cpu().numpy(), v0.double().cpu().numpy() + (k1 + k2) * got.double().cpu().numpy()) < 5e-7


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("channels", [1, 3])
@pytest.mark.parametrize("masked", [False, True])
def test_position_terms(n, channels, masked):
    co, rng, pmid, disp, valid, sp, mesh = _sorted(n, masked, 1)
    field = rng.normal(size=(channels, ) + mesh).astype(np.float32)
    u = rng.normal(size=(n, channels)).astype(np.float32)
    if masked:
        u[~valid] = 0
    f, ud = torch.from_numpy(field).cuda(), torch.from_numpy(u).cuda()
    us = torch.full((n, channels), 9.0, device="cuda")
    dc, ws = sp.interp_grad(f, u=ud, wsum=True, u_sorted=us)
    ref, _ = opm.gather_vjp(pmid, disp, co, field, u, valid=valid)
    bar = 2e-6 * channels * np.abs(u).max() * np.abs(field).max()
    assert np.abs(dc.cpu().numpy() - ref).max() < bar
    refw = opm.gather(pmid, disp, co, field, valid=valid)
    assert np.abs(ws.cpu().numpy() - refw).max() < 2e-6 * np.abs(field).max()
    at = (16 * n + 255) // 256 * 256
    perm = sp.buf[at:at + 4 * n].view(torch.int32).long()
    live = n if valid is None else int(valid.sum())
    assert torch.equal(us[:live], ud[perm[:live]])
    base = torch.from_numpy(rng.normal(size=(n, 3)).astype(np.float32)).cuda()
    acc, _ = sp.interp_grad(f, u=ud, disp_cot=base.clone(), accumulate=True)
    assert torch.equal(acc, base + dc)
    one, _ = sp.interp_grad(f, u=None, u_const=0.5)
    full, _ = sp.interp_grad(f, u=torch.full((n, channels), 0.5, device="cuda"))
    assert torch.equal(one, full)
