"""The ensemble's deposit over its tile shapes, row lengths and remainders: a
member alone in its mesh shape equals the single run bit for bit, whatever the
tile."""
import ctypes

import numpy as np
import pytest
import torch

from tests.test_gpu_ensemble import _members

pytestmark = pytest.mark.gpu

# particles per side, mesh ratio, box, Omega_m: meshes of 6, 10, 14, 44, 50 and 96 cells a side
SPECS = [(6, 1, 30.0, 0.3), (10, 1, 40.0, 0.28), (7, 2, 35.0, 0.3), (11, 4, 50.0, 0.31), (25, 2, 90.0, 0.3),
         (32, 3, 128.0, 0.29)]


@pytest.mark.parametrize("tile", [None, (1, 1), (4, 4), (6, 1), (1, 5), (6, 2)])
def test_tiles_are_bitwise_single_runs(tile):
    import pmpp_b200 as pb
    from pmpp_b200._lib import call
    from pmpp_b200.ensemble import Ensemble
    confs, coss, ics = _members(SPECS, nsteps=2)
    ens = Ensemble(confs, coss)
    if tile is not None:
        shape = (ctypes.c_int32 * len(SPECS))
        call("pmb_ens_set_tiles", ens.handle, shape(*[tile[0]] * len(SPECS)), shape(*[tile[1]] * len(SPECS)))
    outs = ens.forward(ics, graph=False)
    for conf, cos, ic, out in zip(confs, coss, ics, outs):
        ref = pb.NBodyRun(conf, cos).forward(ic)
        for name in ("disp", "vel", "acc"):
            assert torch.equal(getattr(out, name), getattr(ref, name)), (name, conf.mesh_shape)


def test_crowded_member_takes_the_64_bit_sums():
    import pmpp_b200 as pb
    from pmpp_b200.ensemble import Ensemble
    confs, coss, ics = _members([(32, 1, 64.0, 0.3), (16, 2, 64.0, 0.3)], nsteps=2)
    ics[0].disp.copy_((3.2 - ics[0].pmid.float()) * confs[0].cell_size)  # all particles in one cell
    ics[0].vel.zero_()
    outs = Ensemble(confs, coss).forward(ics, graph=False)
    for conf, cos, ic, out in zip(confs, coss, ics, outs):
        ref = pb.NBodyRun(conf, cos).forward(ic)
        assert torch.equal(out.disp, ref.disp) and torch.equal(out.vel, ref.vel)
