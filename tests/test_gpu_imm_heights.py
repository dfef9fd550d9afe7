"""The influence-matrix iteration over wall-normal heights and FD orders at
the edges of its kernels' branches -- each number of rows per lane of the stage
kernel (up to 96, 160, 224, 288 points and beyond), grids lower than a lane's
window, partly filled tiles and solve blocks -- against the oracle, with the
correction written and not, and in place."""

from math import pi

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fd", [2, 4, 6, 8])
@pytest.mark.parametrize("nx,ny,nz", [(16, 11, 16), (12, 65, 24), (16, 159, 8), (8, 161, 16),
                                      (16, 193, 12), (8, 257, 8), (4, 301, 8)])
def test_imm_heights(nx, ny, nz, fd):
    import torch

    from dnsjax_b200 import initial
    from dnsjax_b200.flows.plane_couette import PlaneCouetteFlow
    from dnsjax_b200.parameters import Parameters
    from oracle.config import Config
    from oracle.couette import CouetteSetup

    p = Parameters(phys=dict(system="plane-couette", re=400.0), geo=dict(lx=2 * pi, lz=pi),
                   res=dict(nx=nx, ny=ny, nz=nz, fd_order=fd), step=dict(dt=0.01))
    flow = PlaneCouetteFlow(p)
    imm = {k: v.cpu().numpy() for k, v in flow.imm.items()}
    orc = CouetteSetup(Config(system="plane-couette", nx=nx, ny=ny, nz=nz, lx=2 * pi, lz=pi,
                              re=400.0, dt=0.01, fd_order=fd),
                       imm=dict(imm, D1=flow.D1, D2=flow.D2))
    un, uj, n0, nj = (initial.couette_field(nx, ny, nz, 2 * pi, pi, fd, s, 8.0, 1e-2)
                      for s in (1, 2, 3, 4))
    new, corr = orc.correct(un, uj, n0, nj)
    d = [torch.as_tensor(np.ascontiguousarray(a), device="cuda") for a in (un, uj, n0, nj)]
    got, gcorr = flow.correct(*d)
    # the banded solves' rounding grows with the condition of D2, ~ny^4 eps
    # scaled by dt nu; 1e-12 is met up to 129 points, (301 / 129)^4 = 30 times that at 301
    bound = 1e-12 * max(1.0, (ny / 129.0) ** 4)
    assert rel_l2(got.cpu(), new) < bound
    assert rel_l2(gcorr.cpu(), corr) < bound * np.linalg.norm(new) / np.linalg.norm(corr)
    err = torch.empty(1, dtype=torch.float64, device="cuda")
    fused = flow.correct_fused(*d, err, out=d[1])
    assert bool((fused == got).all())
    assert abs(float(err) - orc.norm(corr)) < bound * orc.norm(new)
    flow.check_status()
