"""The launch count that the bench reports against the profiler: every kernel of the
library (namespace pmb) that the public calls launch, on small and large row counts,
with the FFT pass chain and without."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

pytestmark = pytest.mark.gpu


def _counts(fn):
    from pmpp_b200 import _lib
    fn()  # tables, plans and workspaces
    torch.cuda.synchronize()
    _lib.reset_launch_count()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    seen = [e.name for e in p.events() if e.device_type == torch.autograd.DeviceType.CUDA and "pmb::" in e.name]
    return _lib.launch_count(), seen


def _setup(shape, mesh, dtype="float32"):
    import pmpp_b200 as pb
    conf = pb.Configuration(2.0, shape, mesh, float_dtype=dtype, a_start=0.1, device="cuda")
    p = pb.Particles.gen_grid(conf)
    g = torch.Generator(device="cuda").manual_seed(1)
    p.disp += torch.randn(p.disp.shape, generator=g, device="cuda", dtype=p.disp.dtype)
    return pb, conf, p, pb.SimpleLCDM(conf), torch.randn(p.disp.shape, generator=g, device="cuda", dtype=p.disp.dtype)


@pytest.mark.parametrize("shape,mesh", [((32, 32, 64), 2), ((64, 96, 64), 2), ((32, 384, 64), 2), ((20, 20, 20), 2),
                                        ((90, 100, 8), 2)])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_force_and_adjoint(shape, mesh, dtype):
    pb, conf, p, cos, u = _setup(shape, mesh, dtype)
    for fn in (lambda: pb.gravity(1.0, p, cos, conf), lambda: pb.gravity_vjp(1.0, p, cos, conf, u)):
        n, seen = _counts(fn)
        assert n == len(seen), seen


@pytest.mark.parametrize("shape", [(16, 16, 16), (150, 130, 4)])
def test_particle_mesh_calls(shape):
    pb, conf, p, cos, u = _setup(shape, 1)
    mesh = torch.randn(shape + (3, ), device="cuda")
    modes = torch.fft.rfftn(torch.randn(shape, device="cuda")).contiguous()
    cosb = pb.boltzmann(cos)
    target = np.ones(pb.power_spectrum.num_shells(conf) - 1)
    for fn in (lambda: pb.scatter(p, conf), lambda: pb.scatter(p, conf, val=u), lambda: pb.gather(p, conf, mesh),
               lambda: pb.gather_vjp(p, conf, mesh, u), lambda: pb.scatter(p, conf, cell_size=3.0),
               lambda: pb.scatter(p, conf, val=u, cell_size=3.0), lambda: pb.lpt.lpt(modes, cosb, conf),
               lambda: pb.power_spectrum.pk_loss(p, conf, target)):
        n, seen = _counts(fn)
        assert n == len(seen), seen
