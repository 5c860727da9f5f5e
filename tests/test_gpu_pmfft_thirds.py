"""The FFT pass chain on sides of 3 2^a cells (96 to 768), alone and mixed with
powers of two.

Bars as for the powers of two (test_gpu_pmfft.py): the passes against numpy's
float64 transforms within 1e-5 of the largest value, the force and its adjoint
against the library's transforms within 1e-5, and the chain's stages one by one
against the fused call bit for bit."""
import numpy as np
import pytest
import torch

from tests import test_gpu_pmfft as base
from tests.helpers import random_particles, rel_err

pytestmark = pytest.mark.gpu

SHAPES = [(96, 96, 96), (64, 192, 384), (192, 96, 192), (384, 64, 96), (96, 384, 128), (768, 96, 96), (96, 768, 96),
          (64, 96, 768), (256, 384, 512)]


@pytest.mark.parametrize("shape", SHAPES)
def test_passes_match_numpy(shape):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + 2 * ny + 3 * nz)
    x = rng.normal(size=shape).astype(np.float32)
    got = base._unblock(base._forward(torch.from_numpy(x).cuda(), nx, ny, nz), nx, ny, nz)[0]
    ref = np.fft.rfftn(x.astype(np.float64))
    assert rel_err(base._ri(got), base._ri(ref)) < 1e-5
    X = rng.normal(size=ref.shape) + 1j * rng.normal(size=ref.shape)  # not Hermitian
    out = base._inverse(base._block(X.astype(np.complex64), nx, ny, nz), nx, ny, nz).cpu().numpy()
    assert rel_err(out, np.fft.irfftn(X, s=shape) * (nx * ny * nz)) < 1e-5
    assert base._lib().pmfft_timeouts() == 0


@pytest.mark.parametrize("shape,mesh", [((48, 48, 48), 2), ((96, 96, 96), 1), ((64, 64, 64), 3), ((96, 48, 192), 2),
                                        ((48, 192, 96), 2), ((64, 32, 96), 4), ((16, 16, 128), 6)])
def test_force_and_adjoint_match_library_route_and_stages(shape, mesh):
    from pmpp_b200.runtime import StageTimer
    pb, co, conf = base._confs(shape, mesh)
    assert base._lib().pmfft_active(*conf.mesh_shape)
    pmid, disp = random_particles(co, seed=5, spread=2.0)
    ptcl = pb.Particles(conf, torch.from_numpy(pmid).cuda(), torch.from_numpy(disp).cuda())
    cos = pb.SimpleLCDM(conf)
    ac = torch.from_numpy(np.random.default_rng(2).normal(size=disp.shape).astype(np.float32)).cuda()
    res = {}
    try:
        for on in (True, False):
            base._lib().set_pmfft(on)
            acc = pb.gravity(1.0, ptcl, cos, conf)
            dc, om = pb.gravity_vjp(1.0, ptcl, cos, conf, ac)
            res[on] = (acc, dc, om)
    finally:
        base._lib().set_pmfft(True)
    assert rel_err(res[True][0].cpu().numpy(), res[False][0].cpu().numpy()) < 1e-5
    assert rel_err(res[True][1].cpu().numpy(), res[False][1].cpu().numpy()) < 1e-5
    np.testing.assert_allclose(res[True][2], res[False][2], rtol=1e-5)
    with StageTimer():
        acc = pb.gravity(1.0, ptcl, cos, conf)
        dc, _ = pb.gravity_vjp(1.0, ptcl, cos, conf, ac)
    assert torch.equal(acc, res[True][0]) and torch.equal(dc, res[True][1])
    assert base._lib().pmfft_timeouts() == 0


def test_supported_sides():
    L = base._lib().lib()
    for ok in ((96, 96, 96), (64, 768, 384), (1024, 192, 128)):
        assert L.pmb_pmfft_supported(*ok)
    for no in ((48, 96, 96), (96, 48, 96), (96, 96, 48), (96, 96, 64), (1536, 96, 96), (96, 96, 1536), (160, 96, 96),
               (96, 288, 96)):
        assert not L.pmb_pmfft_supported(*no)
