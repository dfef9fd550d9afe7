"""Every padded length of the two-stage passes on each axis, against the
oracle: the RHS and the transforms, both flow families.  First one length at a
time, the other axes at 16 modes (padded 24, Stockham stages; one column tile of
the periodic flows' y and z passes); then grids of these lengths alone, with
several column tiles of which the last is partly filled, and both block orders of
the curl passes."""

from math import pi

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# mode counts of the lengths beyond 48, 72, 96 and 192 (3 n / 2)
MODES = [24, 36, 72, 96, 108, 144, 192, 256]


def dev(a):
    import torch

    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


# grid of each flow family: several column tiles, a partly filled last one
PERIODIC_GRIDS = [
    (36, 24, 72), (36, 72, 24), (108, 36, 108), (128, 24, 72),
    # a tile's fields next to one another: state and pass buffer beyond 64 MB
    (72, 96, 144),
    (72, 192, 128),  # the same with the 8-column tiles of 288 points
]
COUETTE_GRIDS = [
    (36, 33, 72), (108, 21, 96), (72, 19, 256),
    (144, 65, 144),  # a tile's fields next to one another: beyond 120 MB
    (96, 97, 192),   # the same with 8-column tiles
]


def check_periodic(g, seed):
    from dnsjax_b200 import initial
    from dnsjax_b200.flows.monochromatic import TriplyPeriodicFlow
    from dnsjax_b200.parameters import Parameters
    from oracle.config import Config
    from oracle.fft import spec_to_phys
    from oracle.periodic import PeriodicSetup

    p = Parameters(phys=dict(system="waleffe", re=60.0),
                   geo=dict(lx=2 * pi, lz=2 * pi, tilt_degree=30.0),
                   res=dict(nx=g[0], ny=g[1], nz=g[2]), step=dict(dt=0.01))
    cfg = Config(system="waleffe", nx=g[0], ny=g[1], nz=g[2], lx=2 * pi, lz=2 * pi, ly=2 * pi,
                 re=60.0, dt=0.01, tilt_degree=30.0)
    flow, orc = TriplyPeriodicFlow(p, ly=2 * pi), PeriodicSetup(cfg)
    u0 = initial.periodic_field(*g, 2 * pi, 2 * pi, 2 * pi, seed,
                                initial.kolmogorov_spectrum_k53, 0.1)
    assert rel_l2(flow.get_rhs(dev(u0)).cpu(), orc.get_rhs(u0)) < 1e-12
    phys = spec_to_phys(u0, cfg)
    assert rel_l2(flow.spec_to_phys(dev(u0)).cpu(), phys) < 1e-13
    assert rel_l2(flow.phys_to_spec(dev(phys)).cpu(), u0) < 1e-13


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("n", MODES)
def test_periodic_lengths(n, axis):
    g = [16, 16, 16]
    g[axis] = n
    check_periodic(g, n + axis)


@pytest.mark.parametrize("g", PERIODIC_GRIDS)
def test_periodic_grids(g):
    check_periodic(g, 5)


def check_couette(g, seed):
    from dnsjax_b200 import initial
    from dnsjax_b200.flows.plane_couette import PlaneCouetteFlow
    from dnsjax_b200.parameters import Parameters
    from oracle.config import Config
    from oracle.couette import CouetteSetup
    from oracle.fft import spec_to_phys_2d

    p = Parameters(phys=dict(system="plane-couette", re=400.0), geo=dict(lx=2 * pi, lz=pi),
                   res=dict(nx=g[0], ny=g[1], nz=g[2], fd_order=4), step=dict(dt=0.01))
    cfg = Config(system="plane-couette", nx=g[0], ny=g[1], nz=g[2], lx=2 * pi, lz=pi,
                 re=400.0, dt=0.01, fd_order=4)
    flow = PlaneCouetteFlow(p)
    imm = {k: v.cpu().numpy() for k, v in flow.imm.items()}
    orc = CouetteSetup(cfg, imm=dict(imm, D1=flow.D1, D2=flow.D2))
    u0 = initial.couette_field(*g, 2 * pi, pi, 4, seed, 8.0, 1e-2)
    assert rel_l2(flow.get_rhs(dev(u0)).cpu(), orc.get_rhs(u0)) < 1e-12
    phys = spec_to_phys_2d(u0, cfg)
    assert rel_l2(flow.spec_to_phys(dev(u0)).cpu(), phys) < 1e-13
    assert rel_l2(flow.phys_to_spec(dev(phys)).cpu(), u0) < 1e-13


@pytest.mark.parametrize("axis", [0, 2])
@pytest.mark.parametrize("n", MODES)
def test_couette_lengths(n, axis):
    g = [16, 19, 16]
    g[axis] = n
    check_couette(g, n + axis)


@pytest.mark.parametrize("g", COUETTE_GRIDS)
def test_couette_grids(g):
    check_couette(g, 5)


@pytest.mark.parametrize("system", ["kolmogorov", "plane-couette"])
def test_unrolled_step_graph_lengths(system):
    """Unrolled step graphs on grids of these lengths alone: every kernel of an
    iteration has to honour the skip flag, so the states equal the host loop's
    bit for bit with more iterations unrolled than the step takes."""
    from dnsjax_b200 import driver, initial
    from dnsjax_b200.flows.monochromatic import TriplyPeriodicFlow
    from dnsjax_b200.flows.plane_couette import PlaneCouetteFlow
    from dnsjax_b200.parameters import Parameters

    wall = system == "plane-couette"
    lz = pi if wall else 2 * pi
    p = Parameters(phys=dict(system=system, re=60.0), geo=dict(lx=2 * pi, lz=lz),
                   res=dict(nx=36, ny=33 if wall else 24, nz=72, fd_order=4),
                   step=dict(dt=0.01, corrector_tolerance=1e-10, max_corrector_iterations=60))
    if wall:
        flow = PlaneCouetteFlow(p)
        u0 = initial.couette_field(36, 33, 72, 2 * pi, lz, 4, 1, 8.0, 1e-3)
    else:
        flow = TriplyPeriodicFlow(p, ly=2 * pi)
        u0 = initial.periodic_field(36, 24, 72, 2 * pi, 2 * pi, 2 * pi, 1,
                                    initial.kolmogorov_spectrum_cfg0, 1e-2)
    s_graph, s_host = dev(u0), dev(u0)
    g = flow.make_step_graph(s_graph, unroll=64)
    steppers = flow.make_stepper()
    for _ in range(2):
        s_host, c, e = driver.step(flow, steppers, s_host, 1e-10, 60)
        g.launch()
        assert g.status() == (c, e)
        assert bool((s_graph == s_host).all())


def test_worklist_ensemble_with_192():
    """Work-list ensembles with members that are 192 long on one axis beside
    shorter ones (the wider CTAs of the column kernels): each member's step
    graph's states bit for bit."""
    import torch

    from dnsjax_b200 import initial
    from dnsjax_b200.ensemble import Ensemble
    from dnsjax_b200.flows.monochromatic import TriplyPeriodicFlow
    from dnsjax_b200.parameters import Parameters

    flows, fields = [], []
    for s, g in enumerate([(32, 128, 48), (64, 48, 128), (128, 32, 32), (48, 64, 64)]):
        p = Parameters(phys=dict(system="kolmogorov", re=50.0), geo=dict(lx=2 * pi, lz=2 * pi),
                       res=dict(nx=g[0], ny=g[1], nz=g[2]),
                       step=dict(dt=0.01, corrector_tolerance=1e-10))
        flows.append(TriplyPeriodicFlow(p, ly=2 * pi))
        fields.append(initial.periodic_field(*g, 2 * pi, 2 * pi, 2 * pi, s,
                                             initial.kolmogorov_spectrum_cfg0, 1e-2))
    a = Ensemble(flows, [dev(u) for u in fields], worklist=True)
    b = Ensemble(flows, [dev(u) for u in fields], graphs=True)
    for _ in range(2):
        assert a.step().corrector_iterations == b.step().corrector_iterations
    for x, y in zip(a.states, b.states):
        assert torch.equal(x, y)
    a.close()
    b.close()
