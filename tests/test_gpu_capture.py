"""Calls whose kernels are launched dependent on one another (small grids),
plainly (large ones) and, plane Couette between the two, plainly in the RHS alone,
captured in a CUDA graph by the caller: replays equal the eager calls bit for bit,
alone and back to back.  On the small grids the eager calls also equal those of a
step graph, whose kernels are all launched plainly."""

from math import pi

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system,n", [("kolmogorov", 32), ("kolmogorov", 192),
                                      ("plane-couette", 32), ("plane-couette", 96),
                                      ("plane-couette", 128), ("plane-couette", 144)])
def test_captured_calls(system, n):
    import torch

    from dnsjax_b200.flows.monochromatic import TriplyPeriodicFlow
    from dnsjax_b200.flows.plane_couette import PlaneCouetteFlow
    from dnsjax_b200.parameters import Parameters

    wall = system == "plane-couette"
    p = Parameters(phys=dict(system=system, re=100.0), geo=dict(lx=2 * pi, lz=2 * pi),
                   res=dict(nx=n, ny=n + 1 if wall else n, nz=n, fd_order=4),
                   step=dict(dt=0.01))
    flow = PlaneCouetteFlow(p) if wall else TriplyPeriodicFlow(p, ly=2 * pi)
    g = torch.Generator(device="cuda").manual_seed(n)
    u = torch.view_as_complex(torch.randn(*flow.spec_shape, 2, generator=g,
                                          dtype=torch.float64, device="cuda")) / n**3
    err = torch.empty(1, dtype=torch.float64, device="cuda")

    def calls():
        r = flow.get_rhs(u)
        v = flow.predict(u, r)
        r2 = flow.get_rhs(v)
        return r, r2, flow.correct_fused(u, v, r, r2, err)

    if n == 32:
        pac, _ = flow.make_stepper()
        state = u.clone()
        step = flow.make_step_graph(state, tol=1e30, max_iter=60)  # the first correction
        step.launch()
        assert step.status()[0] == 0
        assert torch.equal(state, flow.correct_velocity(pac(u)[0])[0])
        step.close()
    want = [t.clone() for t in calls()]
    e = err.clone()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = calls()
    for t in got:
        t.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert torch.equal(err, e)
