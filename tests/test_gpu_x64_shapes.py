"""Float64 force, its fused kick and its adjoint on odd, thin and uneven meshes
against the float64 oracle (1e-12 of the largest value, as the cubic ones)."""
import numpy as np
import pytest
import torch

from oracle import pm as opm
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,mesh", [((5, 7, 9), 1), ((3, 4, 2), 2), ((6, 2, 33), 1), ((2, 64, 3), 2),
                                        ((17, 5, 4), 3)])
def test_force_kick_and_adjoint(shape, mesh):
    import pmpp_b200 as pb
    from pmpp_b200 import x64
    co = opm.Conf(2.0, shape, mesh_shape=mesh, float_dtype=np.float64)
    conf = pb.Configuration(2.0, shape, mesh, float_dtype="float64", device="cuda")
    rng = np.random.default_rng(0)
    pmid, disp = opm.gen_grid(co)
    disp = disp + rng.normal(0, 3.0, size=disp.shape)
    vel = rng.normal(size=disp.shape)
    p, d, v = (torch.from_numpy(t).cuda() for t in (pmid, disp, vel))
    acc, _ = x64.force(p, d, conf, 0.3, vel_kick=v, kick=0.25)
    ref = opm.gravity(pmid, disp, co, 0.3)
    assert rel_err(acc.cpu().numpy(), ref) < 1e-12
    assert rel_err(v.cpu().numpy(), vel + 0.25 * ref) < 1e-12
    ac = rng.normal(size=disp.shape)
    cos = pb.SimpleLCDM(conf)
    dc, _ = pb.gravity_vjp(1.0, pb.Particles(conf, p, d), cos, conf, torch.from_numpy(ac).cuda())
    assert rel_err(dc.cpu().numpy(), opm.gravity_vjp(pmid, disp, co, cos.Omega_m, ac)[0]) < 1e-12
