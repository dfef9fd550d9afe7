"""The influence-matrix iteration over wall-normal heights and FD orders at
the edges of its kernels' branches -- each number of rows per lane of the stage
kernel (up to 96, 160, 224, 288 points and beyond), grids lower than a lane's
window, partly filled tiles and solve blocks -- against the oracle, with the
correction written and not, and in place.  Above 160 points the rounding of the
batched substitutions is also held to that of dgbtrs."""

from math import pi

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


GRIDS = [(16, 11, 16), (12, 65, 24), (16, 159, 8), (8, 161, 16), (16, 193, 12), (8, 257, 8),
         (4, 301, 8)]


# 96 x 21 x 128: 192 tiles, beyond the 148 up to which the substitutions of orders 6
# and 8 take one column per lane
@pytest.mark.parametrize("nx,ny,nz,fd", [(*g, fd) for fd in (2, 4, 6, 8) for g in GRIDS]
                         + [(96, 21, 128, 6), (96, 21, 128, 8)])
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


@pytest.mark.parametrize("ny,fd", [(65, 4), (129, 6), (161, 2)])
def test_other_stencils(monkeypatch, ny, fd):
    """D2's even stencils centred half a row the other way: any stencils whose
    rows contain the point are accepted, and these run batched too."""
    import torch

    import dnsjax_b200.fd
    from dnsjax_b200 import _lib, initial
    from dnsjax_b200.flows.plane_couette import PlaneCouetteFlow
    from dnsjax_b200.parameters import Parameters
    from oracle.config import Config
    from oracle.couette import CouetteSetup

    monkeypatch.setattr(dnsjax_b200.fd, "stencil_start",
                        lambda i, n, width: max(0, min(i - (width - 1) // 2, n - width)))
    p = Parameters(phys=dict(system="plane-couette", re=400.0), geo=dict(lx=2 * pi, lz=pi),
                   res=dict(nx=8, ny=ny, nz=8, fd_order=fd), step=dict(dt=0.01))
    flow = PlaneCouetteFlow(p)
    imm = {k: v.cpu().numpy() for k, v in flow.imm.items()}
    orc = CouetteSetup(Config(system="plane-couette", nx=8, ny=ny, nz=8, lx=2 * pi, lz=pi,
                              re=400.0, dt=0.01, fd_order=fd),
                       imm=dict(imm, D1=flow.D1, D2=flow.D2))
    f = [initial.couette_field(8, ny, 8, 2 * pi, pi, fd, s, 8.0, 1e-2) for s in (1, 2, 3, 4)]
    new, _ = orc.correct(*f)
    before = _lib.launch_count()
    got, _ = flow.correct(*[torch.as_tensor(np.ascontiguousarray(a), device="cuda") for a in f])
    assert _lib.launch_count() - before == 5
    assert rel_l2(got.cpu(), new) < 1e-12 * max(1.0, (ny / 129.0) ** 4)
    flow.check_status()


def _fma(a, b, c):
    """a b + c rounded once (an 80-bit product and sum, then 64 bits)."""
    return (np.longdouble(a) * np.longdouble(b) + np.longdouble(c)).astype(np.float64)


def _substitute(ab, piv, kl, b):
    """dgbtrs on columns, multiplying by the diagonal's reciprocal."""
    b, n, d = b.copy(), len(b), 2 * kl
    for j in range(n - 1):
        b[[j, piv[j]]] = b[[piv[j], j]]
        for i in range(1, min(kl, n - 1 - j) + 1):
            b[j + i] = _fma(-ab[d + i, j], b[j], b[j + i])
    for j in range(n - 1, -1, -1):
        b[j] *= 1.0 / ab[d, j]
        for i in range(1, min(d, j) + 1):
            b[j - i] = _fma(-ab[d - i, j], b[j], b[j - i])
    return b


@pytest.mark.parametrize("ny", [193, 257])
def test_tall_substitutions_round_as_dgbtrs(ny):
    """Above 160 points x_j is formed first and multiplies U, as in dgbtrs.  In
    the mean mode grad p cancels the right-hand side, and what is left after one
    update is the rounding of the substitutions: within 1e-4 of the value that
    the same operations give here (measured 5e-5 and 1e-5; the last sums are
    associated differently), 3e-2 and 7e-3 from it with U pre-scaled by its
    diagonal."""
    import torch

    from dnsjax_b200.fd import diff_bands
    from dnsjax_b200.flows.plane_couette import PlaneCouetteFlow
    from dnsjax_b200.parameters import Parameters

    fd = 6
    p = Parameters(phys=dict(system="plane-couette", re=900.0), geo=dict(lx=2 * pi, lz=pi),
                   res=dict(nx=4, ny=ny, nz=4, fd_order=fd), step=dict(dt=0.01))
    flow = PlaneCouetteFlow(p)
    T = np.cos(np.arange(8)[:, None] * np.arccos(np.clip(flow.ys, -1, 1)))
    coef = np.random.default_rng(ny + fd).standard_normal((2, 8)) * np.exp(-1.5 * np.arange(8))
    N = (coef @ T * (1 - flow.ys**2) ** 2).T  # v's right-hand side: re, im
    n = np.zeros(flow.spec_shape, np.complex128)
    n[1, 0, 0] = N[:, 0] + 1j * N[:, 1]
    zero = torch.zeros(flow.spec_shape, dtype=torch.complex128, device="cuda")
    v = flow.predict(zero, torch.as_tensor(n, device="cuda"))[1, 0, 0].cpu().numpy()
    v = np.stack([v.real, v.imag], 1)

    j0, w, _, _ = diff_bands(flow.ys, fd)

    def d1(x):
        out = np.zeros_like(x)
        for m in range(fd + 1):
            out = _fma(w[:, m:m + 1], x[j0 + m], out)
        return out

    imm = {k: a[0, 0].cpu().numpy() for k, a in flow.imm.items()}
    f = d1(N)
    f[[0, -1]] = 0
    R = N - d1(_substitute(imm["Lk_ab"], imm["Lk_piv"], fd, f))
    R[[0, -1]] = 0
    arb = _substitute(imm["Hk_ab"], imm["Hk_piv"], fd, R)
    want = _fma(imm["v2"][:, None], -imm["M_inv"][1, 1] * d1(arb)[-1], arb)
    assert np.linalg.norm(v - want) < 1e-3 * np.linalg.norm(want)
