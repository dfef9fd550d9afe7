"""The work that programs have this package do, as cases to be timed and compared.

Every case calls the public interface of a flow object (``TriplyPeriodicFlow``
or ``PlaneCouetteFlow``) the way a time-stepping or post-processing program
does, on seeded divergence-free fields of the kind the solver advances:

* ``rhs``      the nonlinear term of a state (``get_rhs``), FP64 or, with
               ``fp32``, with the reduced-precision passes of
               ``res.double_precision = False``;
* ``correct``  one corrector update with its norm (``correct_fused``): the
               pointwise update of the periodic flows, the influence-matrix
               iteration of plane Couette;
* ``pac``      ``predict_and_correct`` of the stepper: two right-hand sides,
               the predictor and the first correction;
* ``step``     one whole time step through the step graph, restarted from a
               stored field;
* ``to_phys``, ``to_spec``  the dealiased transforms of snapshots and statistics.

Grids are those of the package's tests, benchmark and workloads (32, 48, 64,
128 modes; 65, 129 wall-normal points) and the sizes between and beyond them
that a user picks: any even mode count whose 3/2 padding is 2^a 3^b, up to
256, and odd wall-normal counts up to 193.

``exact`` is the same mathematics in plain torch: torch.fft transforms, dense
collocation matrices and dense LU solves in 64 bits.
"""

from __future__ import annotations

import math

import numpy as np
import torch

MODES = (24, 32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 256)
FP32_MODES = (32, 48, 64, 128)  # the sizes with reduced-precision passes
COUETTE = "plane-couette"


def _case(op, system, nx, ny, nz, re, dt, **more):
    c = dict(op=op, system=system, nx=nx, ny=ny, nz=nz, re=re, dt=dt, fd=0, tilt=0.0, fp32=False)
    c.update(more)
    return c


def listed():
    def case(name, *args, **more):
        return dict(_case(*args, **more), name=name)

    return [
        # A whole small step: ensembles and parameter studies run thousands of
        # these, and launches and gaps count more than bytes.
        case("kolmogorov32_step", "step", "kolmogorov", 32, 32, 32, 40.0, 0.01),
        # A small decaying box on an uneven grid: prototyping runs.
        case("decaying24x36x48_pac", "pac", "decaying-box", 24, 36, 48, 100.0, 0.01),
        # The benchmark's triply periodic grid, in both precisions.
        case("kolmogorov128_rhs", "rhs", "kolmogorov", 128, 128, 128, 100.0, 0.005),
        case("kolmogorov128_rhs_fp32", "rhs", "kolmogorov", 128, 128, 128, 100.0, 0.005, fp32=True),
        # A tilted shear flow in a stretched box.
        case("waleffe96x72x144_rhs", "rhs", "waleffe", 96, 72, 144, 200.0, 0.01, tilt=24.0),
        # A high-resolution run: the largest case.
        case("kolmogorov256_rhs", "rhs", "kolmogorov", 256, 256, 256, 400.0, 0.002),
        # Reading a snapshot of a mid-size box.
        case("kolmogorov144_to_spec", "to_spec", "kolmogorov", 144, 144, 144, 100.0, 0.005),
        # The middle plane Couette workload: both halves of a first correction.
        case("couette64_pac", "pac", COUETTE, 64, 65, 64, 400.0, 0.02, fd=4),
        # The benchmark's plane Couette grid: the two halves of an iteration.
        case("couette128_rhs", "rhs", COUETTE, 128, 129, 128, 1000.0, 0.01, fd=6),
        case("couette128_correct", "correct", COUETTE, 128, 129, 128, 1000.0, 0.01, fd=6),
        # Wall resolution above the benchmark's on an uneven grid.
        case("couette96x193x72_pac", "pac", COUETTE, 96, 193, 72, 2000.0, 0.005, fd=4),
        # Physical fields for statistics and snapshots.
        case("couette128_to_phys", "to_phys", COUETTE, 128, 129, 128, 1000.0, 0.01, fd=6),
    ]


def draw(rng):
    op = rng.choice(("rhs", "rhs", "rhs", "rhs", "correct", "correct", "pac", "pac", "step", "to_phys", "to_spec"))
    couette = rng.random() < 0.5
    fp32 = op in ("rhs", "pac") and rng.random() < 0.3
    sizes = FP32_MODES if fp32 else MODES
    # grid points of the largest drawn case, by what a pass of the op runs
    top = {"rhs": 256, "to_phys": 256, "to_spec": 256, "correct": 256, "pac": 192, "step": 72}[op] ** 3
    if couette:
        top = min(top, 128 * 128 * 193)
    while True:
        g = math.exp(rng.uniform(math.log(24), math.log(256)))

        nx, ny, nz = (g * math.exp(rng.uniform(-0.5, 0.5)) for _ in range(3))
        nx, nz = (min(sizes, key=lambda n: abs(math.log(n / v))) for v in (nx, nz))  # noqa: B023
        # any odd count of wall-normal points
        ny = min(193, max(33, int(ny) | 1)) if couette else min(sizes, key=lambda n: abs(math.log(n / ny)))
        if nx * ny * nz <= top:
            break
    if couette:
        return _case(op, COUETTE, nx, ny, nz, float(round(math.exp(rng.uniform(math.log(200), math.log(2000))))),
                     0.01, fd=rng.choice((4, 6)), fp32=fp32)
    return _case(op, rng.choice(("kolmogorov", "waleffe", "decaying-box")), nx, ny, nz,
                 float(round(math.exp(rng.uniform(math.log(40), math.log(400))))), 0.005,
                 tilt=rng.choice((0.0, 0.0, 24.0, 90.0)), fp32=fp32)


TOL, CAP = 1e-10, 60  # corrector tolerance and iteration cap of the step cases


def _box(c):
    """(lx, ly, lz)"""
    return (2 * math.pi, 2.0, math.pi) if c["system"] == COUETTE else (2 * math.pi,) * 3


def _flow(c):
    from dnsjax_b200.flows.monochromatic import TriplyPeriodicFlow
    from dnsjax_b200.flows.plane_couette import PlaneCouetteFlow
    from dnsjax_b200.parameters import Parameters

    lx, ly, lz = _box(c)
    res = dict(nx=c["nx"], ny=c["ny"], nz=c["nz"], double_precision=not c["fp32"])
    if c["fd"]:
        res["fd_order"] = c["fd"]
    p = Parameters(phys=dict(system=c["system"], re=c["re"]), geo=dict(lx=lx, lz=lz, tilt_degree=c["tilt"]), res=res,
                   step=dict(dt=c["dt"], corrector_tolerance=TOL, max_corrector_iterations=CAP))
    return PlaneCouetteFlow(p) if c["system"] == COUETTE else TriplyPeriodicFlow(p, ly=ly)


def prepare(case, seed):
    flow = _flow(case)
    st = {"op": case["op"], "flow": flow}
    u = _field(case, seed)
    op = case["op"]
    if op in ("rhs", "to_phys"):
        st["u"] = u
    elif op == "to_spec":
        st["phys"] = _to_phys(case, u).contiguous()
    elif op == "pac":
        st["u"] = u
        st["pac"] = flow.make_stepper()[0]
    elif op == "correct":
        st["args"] = _iterate(case, seed, u)
        st["err"] = torch.empty(1, dtype=torch.float64, device=u.device)
    else:
        st["u"], st["state"] = u, u.clone()
        st["graph"] = flow.make_step_graph(st["state"])
    return st


def run(st):
    op, flow = st["op"], st["flow"]
    if op == "rhs":
        return flow.get_rhs(st["u"])
    if op == "correct":
        return flow.correct_fused(*st["args"], st["err"]), st["err"]
    if op == "pac":
        return st["pac"](st["u"])
    if op == "to_phys":
        return flow.spec_to_phys(st["u"])
    if op == "to_spec":
        return flow.phys_to_spec(st["phys"])
    st["state"].copy_(st["u"])
    st["graph"].launch()
    return st["state"]


def _counts(c):
    """(spectral points of one component, padded points, FFT flops of one field)"""
    nkx, nz1 = c["nx"] // 2, c["nz"] - 1
    mx, mz = 3 * c["nx"] // 2, 3 * c["nz"] // 2
    fft = lambda m: 5.0 * m * math.log2(m)  # noqa: E731
    if c["system"] == COUETTE:
        my, s, f = c["ny"], c["ny"] * nz1 * nkx, 0.0
    else:
        my = 3 * c["ny"] // 2
        s, f = (c["ny"] - 1) * nz1 * nkx, fft(my) * nz1 * nkx
    return s, mx * my * mz, f + fft(mz) * my * nkx + 0.5 * fft(mx) * my * mz


def work(case):
    s, points, fft = _counts(case)
    field = 3 * s * 16.0
    rhs = {"bytes": 2 * field, "flops": 9 * fft + 40.0 * points}
    if case["system"] == COUETTE:
        p = case["fd"]
        # u^n, u^j, N^n, N^j in, u^{j+1} out; the factors of L_k and H_k (p
        # multipliers and p + 2 of U a row, shared by the modes +-kz) and v1, v2, q1, q2
        cor = {"bytes": 5 * field + s * 8.0 * ((2 * p + 2) + 4),
               "flops": s * (8 * 2 * (2.0 * p + (2 * p + 4)) + 2 * 2.0 * (7 * (p + 1) + 4 * (p + 2)) + 80)}
    else:
        cor = {"bytes": 4 * field + s * 8.0, "flops": 24.0 * s}
    op = case["op"]
    if op == "rhs":
        n = (1, 0)
    elif op == "correct":
        n = (0, 1)
    elif op in ("to_phys", "to_spec"):
        return {"bytes": field + 3 * 8.0 * points, "flops": 3 * fft}
    else:
        n = (2, 2) if op == "pac" else (5, 5)  # a step: the first correction and about three more
    return {k: n[0] * rhs[k] + n[1] * cor[k] for k in ("bytes", "flops")}


def tolerance(case):
    """About four times the relative errors seen against ``exact``: 9e-16 for
    the transforms, 3e-7 in 32 bits, 4e-14 (grids up to 128 x 129 x 128) to
    2e-13 where L_k, whose condition grows with the wall-normal points, is solved."""
    if case["fp32"]:
        return {"rel": 1e-6, "max": 4e-5}
    if case["op"] == "step":  # the iteration stops at TOL: a result may be one iteration from another's
        return {"rel": 1e-9, "max": 1e-7}
    if case["system"] == COUETTE and case["op"] in ("pac", "correct"):
        return {"rel": 1e-12, "max": 1e-10}
    return {"rel": 5e-15, "max": 5e-13}


# -- the same mathematics in plain torch -----------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _harmonics(n):
    """Stored harmonics of a complex axis: FFT order without the Nyquist mode."""
    q = np.fft.fftfreq(n, 1.0 / n)
    return np.delete(q, n // 2)


def _k(c):
    """(kx, ky, kz) shaped for a component of a state; ky is None for plane Couette."""
    lx, ly, lz = _box(c)
    t = lambda a, shape: torch.tensor(a, dtype=torch.float64, device=_device()).reshape(shape)  # noqa: E731
    kx = 2 * math.pi / lx * np.arange(c["nx"] // 2)
    kz = 2 * math.pi / lz * _harmonics(c["nz"])
    if c["system"] == COUETTE:
        return t(kx, (1, -1, 1)), None, t(kz, (-1, 1, 1))
    return t(kx, (1, 1, -1)), t(2 * math.pi / ly * _harmonics(c["ny"]), (-1, 1, 1)), t(kz, (1, -1, 1))


def _mirror(a, dims):
    """a(-k) along Nyquist-free axes."""
    for d in dims:
        a = torch.cat([a.narrow(d, 0, 1), a.narrow(d, 1, a.size(d) - 1).flip(d)], d)
    return a


def _normal(c, seed, shape):
    g = torch.Generator(device=_device()).manual_seed(int(seed))
    return torch.view_as_complex(torch.randn(*shape, 2, generator=g, dtype=torch.float64, device=_device()))


def _hermitian(c, u):
    """The kx = 0 plane of a real field."""
    d, kz_dim = (2, 1) if c["system"] == COUETTE else (3, 2)
    plane = u.select(d, 0)
    dims = [kz_dim] if c["system"] == COUETTE else [1, 2]
    plane.copy_(0.5 * (plane + _mirror(plane, dims).conj()))
    return u


def _field(c, seed, stretch=1.0):
    """A divergence-free perturbation: k^-5/3 with a Gaussian cut-off near the
    grid's own (periodic), the curl of a wall-bounded potential (Couette)."""
    kx, ky, kz = _k(c)
    if c["system"] == COUETTE:
        y, D1, _ = _matrices(c)
        shape = (3, c["nz"] - 1, c["nx"] // 2, c["ny"])
        cut = (min(c["nx"], c["nz"]) / 8.0) ** 2
        coef = _normal(c, seed, shape[:3] + (4,))
        cheb = torch.stack([torch.cos(m * torch.arccos(y.clamp(-1, 1))) for m in range(4)]).to(coef.dtype)
        psi = (coef @ cheb) * ((1 - y**2) ** 2) * torch.exp(-stretch * (kx**2 + kz**2) / cut)
        d = psi @ D1.T.to(psi.dtype)
        u = torch.stack([d[2] - 1j * kz * psi[1], 1j * kz * psi[0] - 1j * kx * psi[2], 1j * kx * psi[1] - d[0]])
        u[..., 0] = 0
        u[..., -1] = 0
        weight = torch.where(kx == 0, 1.0, 2.0)
        e = float(((u.abs() ** 2).sum(0) * weight * _simpson(y)).sum()) / 4
        return _hermitian(c, u * math.sqrt(0.05 / e)).contiguous()
    k2 = kx**2 + ky**2 + kz**2
    cut = (min(c["nx"], c["ny"], c["nz"]) / 6.0) ** 2
    amp = torch.where(k2 > 0, k2.clamp_min(1e-30) ** (-5.0 / 6.0), 0.0) * torch.exp(-stretch * k2 / cut)
    u = _hermitian(c, _normal(c, seed, (3,) + tuple(k2.shape)) * amp)
    div = (kx * u[0] + ky * u[1] + kz * u[2]) / torch.where(k2 > 0, k2, 1.0)
    u = torch.stack([u[0] - kx * div, u[1] - ky * div, u[2] - kz * div])
    weight = torch.where(kx == 0, 1.0, 2.0)
    e = float(((u.abs() ** 2).sum(0) * weight).sum()) / 2
    return (u * math.sqrt((0.01 if c["nx"] <= 64 else 0.5) / e)).contiguous()


def _pad(a, m, dim):
    h = (a.size(dim) + 1) // 2
    shape = list(a.shape)
    shape[dim] = m
    out = a.new_zeros(shape)
    out.narrow(dim, 0, h).copy_(a.narrow(dim, 0, h))
    out.narrow(dim, m - h + 1, h - 1).copy_(a.narrow(dim, h, h - 1))
    return out


def _cut(a, n, dim):
    h, m = n // 2, a.size(dim)
    return torch.cat([a.narrow(dim, 0, h), a.narrow(dim, m - h + 1, h - 1)], dim)


def _to_phys(c, u):
    mx, mz = 3 * c["nx"] // 2, 3 * c["nz"] // 2
    out = []
    for f in u:  # a field at a time
        if c["system"] == COUETTE:
            f = torch.fft.ifft(_pad(f, mz, 0), dim=0, norm="forward")
            out.append(torch.fft.irfft(f, n=mx, dim=1, norm="forward").permute(2, 0, 1))
        else:
            f = torch.fft.ifft(_pad(f, 3 * c["ny"] // 2, 0), dim=0, norm="forward")
            f = torch.fft.ifft(_pad(f, mz, 1), dim=1, norm="forward")
            out.append(torch.fft.irfft(f, n=mx, dim=2, norm="forward"))
    return torch.stack(out)


def _to_spec(c, v):
    out = []
    for f in v:
        f = torch.fft.rfft(f, dim=2, norm="forward")[..., : c["nx"] // 2]
        f = _cut(torch.fft.fft(f, dim=1, norm="forward"), c["nz"], 1)
        if c["system"] == COUETTE:
            out.append(f.permute(1, 2, 0).contiguous())
        else:
            out.append(_cut(torch.fft.fft(f, dim=0, norm="forward"), c["ny"], 0))
    return torch.stack(out)


def _base(c):
    """Base flow, its curl and U x curl U at the physical y points, [3][y]."""
    if c["system"] == COUETTE:
        y = _matrices(c)[0]
        zero, one = torch.zeros_like(y), torch.ones_like(y)
        return torch.stack([y, zero, zero]), torch.stack([zero, zero, -one]), torch.stack([zero, y, zero])
    n, a = 3 * c["ny"] // 2, 2 * math.pi / _box(c)[1]
    x = torch.arange(n, dtype=torch.float64, device=_device()) * (2 * math.pi / n)
    zero = torch.zeros_like(x)
    if c["system"] == "decaying-box":
        U, dU = zero, zero
    elif c["system"] == "kolmogorov":
        U, dU = torch.sin(x), a * torch.cos(x)
    else:
        U, dU = torch.cos(x), -a * torch.sin(x)
    co, si = math.cos(math.radians(c["tilt"])), math.sin(math.radians(c["tilt"]))
    return (torch.stack([co * U, zero, si * U]), torch.stack([si * dU, zero, -co * dU]),
            torch.stack([zero, U * dU, zero]))


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _rhs(c, u):
    kx, ky, kz = _k(c)
    if c["system"] == COUETTE:
        D1 = _matrices(c)[1].T.to(u.dtype)
        w = torch.stack([u[2] @ D1 - 1j * kz * u[1], 1j * kz * u[0] - 1j * kx * u[2], 1j * kx * u[1] - u[0] @ D1])
    else:
        w = 1j * torch.stack([ky * u[2] - kz * u[1], kz * u[0] - kx * u[2], kx * u[1] - ky * u[0]])
    U, cU, nU = (b[:, :, None, None] for b in _base(c))
    v, w = _to_phys(c, u), _to_phys(c, w)
    n = _to_spec(c, _cross(v, w) + _cross(v, cU.expand_as(v)) + _cross(U.expand_as(v), w) + nU)
    if c["system"] == COUETTE:
        return n
    k2 = kx**2 + ky**2 + kz**2
    div = (kx * n[0] + ky * n[1] + kz * n[2]) / torch.where(k2 > 0, k2, 1.0)
    return torch.stack([n[0] - kx * div, n[1] - ky * div, n[2] - kz * div])


def _matrices(c):
    """(y, D1, D2) on the Chebyshev-Gauss-Lobatto points: derivatives at a node
    of the polynomial through the fd + 1 (fd + 2) nodes around it, by the
    barycentric formulas (Welfert 1997)."""
    n, p = c["ny"], c["fd"]
    y64 = -np.cos(np.arange(n, dtype=np.float64) * np.pi / (n - 1))
    y = y64.astype(np.longdouble)
    mats = []
    for width, order in ((p + 1, 1), (p + 2, 2)):
        D = np.zeros((n, n))
        for i in range(n):
            j0 = max(0, min(i - width // 2, n - width))
            x, me = y[j0:j0 + width], i - j0
            gap = x[:, None] - x[None, :]
            np.fill_diagonal(gap, 1)
            w = 1 / gap.prod(1)
            d = np.delete(gap[me], me)  # x_i - x_j
            r1 = np.delete(w, me) / w[me] / d
            row = r1 if order == 1 else 2 * r1 * (-r1.sum() - 1 / d)
            row = np.insert(row, me, -row.sum())
            D[i, j0:j0 + width] = row.astype(np.float64)
        mats.append(D)
    return tuple(torch.tensor(a, dtype=torch.float64, device=_device()) for a in (y64, *mats))


def _simpson(y):
    w = torch.zeros_like(y)
    h = y[1:] - y[:-1]
    h0, h1 = h[:-1:2], h[1::2]
    s = h0 + h1
    w[:-2:2] += s / 6 * (2 - h1 / h0)
    w[1:-1:2] += s / 6 * s**2 / (h0 * h1)
    w[2::2] += s / 6 * (2 - h0 / h1)
    return w


def _influence(c, un, uj, Nn, Nj):
    """One influence-matrix iteration -> u^{j+1}, by dense solves a kz plane group at a time."""
    y, D1, D2 = _matrices(c)
    kx, _, kz = _k(c)
    ny, dt, th, nu = c["ny"], c["dt"], 0.5, 1.0 / c["re"]
    eye = torch.eye(ny, dtype=torch.float64, device=y.device)
    new = torch.empty_like(un)
    step = max(1, int(2e8 // (kx.numel() * ny * ny)))
    real = lambda z: torch.view_as_real(z)  # noqa: E731  (..., ny, 2)
    for s in range(0, kz.numel(), step):
        b = slice(s, min(s + step, kz.numel()))
        kzb = kz[b]
        k2 = (kx**2 + kzb**2)[..., 0]
        zero = k2 == 0
        A = D2 - k2[..., None, None] * eye
        Dt = D1.T.to(un.dtype)
        div = lambda q: 1j * kx * q[0] + q[1] @ Dt + 1j * kzb * q[2]  # noqa: E731, B023
        u, n0, nj = un[:, b], Nn[:, b], Nj[:, b]
        d = div(u)
        f = d / dt + th * div(nj) + (1 - th) * div(n0) + (1 - th) * nu * (d @ D2.T.to(d.dtype) - k2[..., None] * d)
        L = A.clone()
        L[..., 0, :] = torch.where(zero[..., None], eye[0], D1[0])
        L[..., -1, :] = D1[-1]
        ends = torch.stack([eye[0], eye[-1]], 1).expand(*k2.shape, ny, 2)
        f[..., 0] = 0
        f[..., -1] = 0
        sol = torch.linalg.solve(L, torch.cat([real(f), ends], -1))
        p, P12 = torch.view_as_complex(sol[..., :2].contiguous()), sol[..., 2:]
        H = eye / dt - th * nu * A
        for w in (0, -1):
            H[..., w, :] = eye[w]
        grad = torch.stack([1j * kx * p, p @ Dt, 1j * kzb * p])
        R = u / dt + (1 - th) * nu * (u @ D2.T.to(u.dtype) - k2[..., None] * u) - grad + th * nj + (1 - th) * n0
        cols = torch.cat([real(R[0]), real(R[1]), real(R[2]), -(D1 @ P12), P12], -1)
        cols[..., 0, :] = 0
        cols[..., -1, :] = 0
        sol = torch.linalg.solve(H, cols)
        arb = [torch.view_as_complex(sol[..., 2 * i:2 * i + 2].contiguous()) for i in range(3)]
        V, Q = sol[..., 6:8], sol[..., 8:10]
        walls = D1[[0, -1]]
        M = walls @ V
        rhs = -(walls.to(un.dtype) @ arb[1][..., None])  # (..., 2, 1)
        # the mean mode: only the upper wall's condition is left
        M = torch.where(zero[..., None, None], torch.stack([torch.stack([torch.ones_like(k2), torch.zeros_like(k2)], -1),
                                                            torch.stack([torch.zeros_like(k2), M[..., 1, 1]], -1)], -2), M)
        rhs[..., 0, 0] = torch.where(zero, 0, rhs[..., 0, 0])
        a = torch.linalg.solve(M, real(rhs[..., 0]))
        a = torch.view_as_complex(a.contiguous())[..., None]
        q = (Q.to(a.dtype) @ a)[..., 0]
        new[0, b] = arb[0] - 1j * kx * q
        new[1, b] = arb[1] + (V.to(a.dtype) @ a)[..., 0]
        new[2, b] = arb[2] - 1j * kzb * q
    return new


def _norm(c, v):
    kx = _k(c)[0]
    e = (v.abs() ** 2).sum(0) * torch.where(kx == 0, 1.0, 2.0)
    if c["system"] == COUETTE:
        e = e * _simpson(_matrices(c)[0]) / _box(c)[1]
    return e.sum().sqrt().reshape(1)


def _helmholtz(c):
    """Crank-Nicolson coefficients of the periodic flows, the mean mode's zero."""
    kx, ky, kz = _k(c)
    k2 = kx**2 + ky**2 + kz**2
    l1 = 1 / c["dt"] - 0.5 * k2 / c["re"]
    l2 = 1 / (1 / c["dt"] + 0.5 * k2 / c["re"])
    return torch.where(k2 == 0, 0.0, l1), torch.where(k2 == 0, 0.0, l2)


def _predict(c, u, N):
    if c["system"] == COUETTE:
        return _influence(c, u, u, N, N)
    l1, l2 = _helmholtz(c)
    return (u * l1 + N) * l2


def _correct(c, u, pred, prev, nxt):
    if c["system"] == COUETTE:
        new = _influence(c, u, pred, prev, nxt)
        return new, _norm(c, new - pred)
    corr = 0.5 * (nxt - prev) * _helmholtz(c)[1]
    return pred + corr, _norm(c, corr)


def _iterate(c, seed, u):
    """A corrector's arguments: the state, an iterate near it and the two right-hand sides."""
    v = u + 0.02 * _field(c, int(seed) + 7919, 1.5)
    return [u, v, _rhs(c, u), _rhs(c, v)]


def exact(case, seed):
    c = case
    u = _field(c, seed)
    op = c["op"]
    if op == "rhs":
        return _rhs(c, u)
    if op == "to_phys":
        return _to_phys(c, u)
    if op == "to_spec":
        return _to_spec(c, _to_phys(c, u))
    if op == "correct":
        return _correct(c, *_iterate(c, seed, u))
    prev = _rhs(c, u)
    v = _predict(c, u, prev)
    nxt = _rhs(c, v)
    v, err = _correct(c, u, v, prev, nxt)
    if op == "pac":
        return v, nxt, err
    for _ in range(CAP):
        if not float(err) > TOL:
            break
        prev, nxt = nxt, _rhs(c, v)
        v, err = _correct(c, u, v, prev, nxt)
    if c["system"] != COUETTE:
        kx, ky, kz = _k(c)
        k2 = kx**2 + ky**2 + kz**2
        div = (kx * v[0] + ky * v[1] + kz * v[2]) / torch.where(k2 > 0, k2, 1.0)
        v = torch.stack([v[0] - kx * div, v[1] - ky * div, v[2] - kz * div])
        v[:, 0, 0, 0] = 0
    return v
