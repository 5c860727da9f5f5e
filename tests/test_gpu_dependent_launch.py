"""Kernels that may start before the one ahead of them has ended (meshes of up to
2^23 cells) and plain launches above: forces and adjoints of alternating states
issued without a synchronisation, on two streams and captured in a graph, equal
the ones with a synchronisation after each, bit for bit."""
import numpy as np
import pytest
import torch

from oracle import pm as opm
from tests.helpers import random_particles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,mesh", [((32, 32, 64), 2), ((24, 20, 18), 2), ((64, 128, 128), 2), ((48, 96, 256), 2),
                                        ((64, 128, 192), 2)])
def test_unsynchronised_calls_bitwise(shape, mesh):
    import pmpp_b200 as pb
    co = opm.Conf(2.0, shape, mesh_shape=mesh)
    conf = pb.Configuration(2.0, shape, mesh, device="cuda")
    cos = pb.SimpleLCDM(conf)
    sets = []
    for seed in range(3):
        pmid, disp = random_particles(co, seed=seed, spread=2.0 + seed)
        u = np.random.default_rng(seed).normal(size=disp.shape).astype(np.float32)
        sets.append((pb.Particles(conf, torch.from_numpy(pmid).cuda(), torch.from_numpy(disp).cuda()),
                     torch.from_numpy(u).cuda()))

    def both(k):
        p, u = sets[k]
        return pb.gravity(1.0, p, cos, conf), pb.gravity_vjp(1.0, p, cos, conf, u)[0]

    ref = []
    for k in range(3):
        ref.append(both(k))
        torch.cuda.synchronize()
    got = [pb.gravity(1.0, sets[i % 3][0], cos, conf) for i in range(12)] + [both(i % 3) for i in range(6)]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        other = [pb.gravity(1.0, sets[i % 3][0], cos, conf) for i in range(6)]
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        held = [pb.gravity(1.0, sets[k][0], cos, conf) for k in range(3)]
    for h in held:
        h.zero_()
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    for i in range(12):
        assert torch.equal(got[i], ref[i % 3][0])
    for i in range(6):
        assert torch.equal(got[12 + i][0], ref[i % 3][0]) and torch.equal(got[12 + i][1], ref[i % 3][1])
        assert torch.equal(other[i], ref[i % 3][0])
    for k in range(3):
        assert torch.equal(held[k], ref[k][0])


@pytest.mark.parametrize("mesh,n", [((16, 16, 16), 1 << 17), ((16, 16, 16), 1 << 18), ((32, 8, 64), 300000),
                                    ((8, 8, 8), 200000)])
def test_crowded_small_mesh_bitwise(mesh, n):
    """Deposits of many particles on few rows, early and plain, right after their sort and before a gather
    of what they wrote: no synchronisation in between against one after each."""
    import pmpp_b200 as pb
    from pmpp_b200.cic import SortedParticles
    conf = pb.Configuration(2.0, mesh, 1, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(2)
    side = torch.tensor(mesh, device="cuda")
    sets = [((torch.rand((n, 3), generator=g, device="cuda") * side).to(torch.int16),
             torch.randn((n, 3), generator=g, device="cuda")) for _ in range(2)]

    def run(k, sync):
        wait = torch.cuda.synchronize if sync else lambda: None
        sp = SortedParticles(*sets[k], conf)
        wait()
        rho = sp.scatter(val_const=0.25)
        wait()
        return rho, sp.gather(rho.expand(3, *mesh).contiguous())

    ref = [run(k, True) for k in range(2)]
    got = [run(i % 2, False) for i in range(8)]
    for i, (rho, v) in enumerate(got):
        assert torch.equal(rho, ref[i % 2][0]) and torch.equal(v, ref[i % 2][1])
