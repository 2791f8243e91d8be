"""The work whose speed this framework is judged by: forward models,
sensitivities, Gauss-Newton steps, inner solves and batches of complex
resistivity surveys, through the public entry points (lib.Context, lib.Batch).

A case names a kind of call, a mesh (quadrilaterals or split quadrilaterals,
with or without topography, mixed or Dirichlet sides), the electrodes and the
dipole-dipole readings on it.  listed() spans the sizes of the repository's own
configurations: 480 to 60,160 cells, 10 to 128 electrodes, 42 to about 12,000
readings.  The seed gives the ground (layers and blocks of complex resistivity)
and the noise of the data.  exact() restates the finite-element model, the
sensitivities and the inner solves in plain 64-bit torch.
"""
import functools
import math

import numpy as np
import torch

from crtomo_stable_b200 import regularization, synth
from crtomo_stable_b200.lib import PREC_FP64, PREC_MIXED, PRECOND_BLOCK, PRECOND_JACOBI, Batch, Context

CASE = dict(kind="forward", nx=60, nz=20, nel=40, tri=False, topo=False, dirichlet=False, dc=False, mixed=False,
            spacings=1, nmax=8, gradient=False, block=False, lam=1.0, count=1)


def case(**kw):
    return {**CASE, **kw}


def listed():
    return [
        # one CRMod run of a small field line: 60 x 20 quadrilaterals, 40 electrodes, responses times the
        # geometric factor
        case(name="forward-40el"),
        # CRMod with the sensitivity files: a small profile, sens(nanz, elanz) copied to the host
        case(name="sens-10el", kind="sens", nx=44, nz=16, nel=10, nmax=6),
        # real (DC) forward of a long profile with topography
        case(name="forward-dc-96el", nx=180, nz=36, nel=96, tri=True, topo=True, dc=True, spacings=2, nmax=10),
        # a mesh that is cut off by Dirichlet sides: one factor per wavenumber, complex64 with refinement
        case(name="forward-dirichlet", nx=100, nz=40, nel=48, dirichlet=True, mixed=True, spacings=2, nmax=8),
        # the trial models of a line search: 20,000 quadrilaterals, 96 electrodes, complex128
        case(name="forward-20k", nx=200, nz=100, nel=96, spacings=4, nmax=12),
        # the start of an inversion: response, sensitivities, lambda_0 and coverage on 8,000 triangles with
        # topography
        case(name="start-48el", kind="start", nx=100, nz=40, nel=48, tri=True, topo=True, mixed=True, spacings=2,
             nmax=10),
        # a Gauss-Newton step where latency counts: 480 triangles, 12 electrodes, the reference's CG
        case(name="gn-12el", kind="gn", nx=24, nz=10, nel=12, tri=True, topo=True, spacings=2, nmax=4),
        # a DC Gauss-Newton step (real Jacobian) on 8,000 triangles
        case(name="gn-dc-48el", kind="gn", nx=100, nz=40, nel=48, tri=True, dc=True, spacings=2, nmax=10,
             block=True),
        # the benchmark's Gauss-Newton step: 60,160 triangles, 128 electrodes, dipole-dipole and gradient readings
        case(name="gn-60k", kind="gn", nx=235, nz=128, nel=128, tri=True, mixed=True, spacings=10, nmax=10,
             gradient=True, block=True),
        # one model update with the reference's CG on a Jacobian that the caller holds, complex128
        case(name="update-9600", kind="update", nx=160, nz=60, nel=64, spacings=3, nmax=8),
        # the lambda trials of one iterate side by side, complex64 Jacobian
        case(name="trials-9600", kind="trials", nx=120, nz=40, nel=64, tri=True, mixed=True, spacings=3, nmax=10,
             count=4),
        # independent surveys of uneven size in one batch (forward and sensitivities under one graph)
        case(name="batch-12", kind="batch", nx=110, nz=40, nel=64, tri=True, mixed=True, count=12),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["forward", "forward", "sens", "start", "gn", "gn", "update", "trials", "batch"])
    tri = rng.random() < 0.6
    c = case(kind=kind, tri=tri, topo=tri and rng.random() < 0.5, spacings=rng.randint(1, 4),
             nmax=rng.randint(4, 12), dc=rng.random() < 0.3, mixed=rng.random() < 0.6)
    c["nz"] = logint(10, 120)
    c["nx"] = logint(24, 200)
    if kind == "sens":
        c.update(nx=logint(24, 70), nz=logint(10, 24), mixed=False, dc=False, spacings=1)
    if kind in ("update", "trials"):
        c.update(nx=logint(24, 160), nz=logint(10, 60), dc=False, lam=10.0 ** rng.uniform(-1, 1))
    if kind == "trials":
        c["count"] = rng.randint(2, 8)
    if kind == "batch":
        c.update(tri=True, topo=False, mixed=True, dc=False, count=rng.randint(2, 12), nx=logint(40, 110),
                 nz=logint(10, 40))
    if kind == "forward":
        c["dirichlet"] = rng.random() < 0.3
    if kind == "gn":
        c["block"] = True
        c["lam"] = 10.0 ** rng.uniform(-1, 1)
    c["nel"] = min(logint(10, 128), c["nx"] - 10)
    return c


# -- the survey ---------------------------------------------------------------

def frozen(c):
    return tuple(sorted((k, v) for k, v in c.items() if k != "name"))


@functools.lru_cache(maxsize=64)
def survey(key):
    """Mesh, electrodes, readings and regulariser of a case: what stays the same while the ground changes."""
    c = dict(key)
    nx, nz, nel = c["nx"], c["nz"], c["nel"]
    xs = np.arange(nx + 1, dtype=np.float64) - (nx - nel) // 2
    depths = synth.graded_depths(nz, 0.25 if nz > 24 else 0.5, 1.0 + 3.5 / nz)
    topo = (lambda x: np.sin(2 * np.pi * x / 20.0)) if c["topo"] else None
    mesh = synth.structured_mesh(xs, depths, triangles=c["tri"], topo=topo, side_type=13 if c["dirichlet"] else 11)
    enr = synth.surface_electrodes(mesh, xs, np.arange(nel, dtype=np.float64), nz)
    configs = synth.dipole_dipole(nel, tuple(range(1, c["spacings"] + 1)), c["nmax"])
    if c["gradient"]:
        for span, step in ((nel // 4, 2), (nel // 2, 4), (3 * nel // 8, 4)):
            configs += synth.gradient(nel, span, step)
    strnr, vnr = synth.encode(configs)
    reg = None
    if c["kind"] in ("gn", "update", "trials"):
        if c["tri"]:
            nb = regularization.nachbar(mesh)
            reg = dict(ltri=1, smatm=regularization.smatm_tri(mesh, nb, 1.0, 1.0), nachbar=nb)
        else:
            reg = dict(ltri=0, smatm=regularization.smatm_reg(mesh, nx, nz, 1.0, 1.0), nx=nx)
    return mesh, enr, strnr, vnr, reg


def ground(mesh, rng):
    """Layers and blocks: complex conductivity per cell, 10 to 1000 Ohm m and -1 to -30 mrad."""
    cx, cy = synth.centroids(mesh)
    depth = -cy
    rho = np.full(mesh.elanz, math.exp(rng.uniform(math.log(20), math.log(500))))
    pha = np.full(mesh.elanz, -rng.uniform(1, 30))
    for b in sorted(rng.uniform(2.0, 0.7 * depth.max(), 2)):
        rho[depth > b] = math.exp(rng.uniform(math.log(20), math.log(500)))
        pha[depth > b] = -rng.uniform(1, 30)
    for _ in range(3):
        x0, z0 = rng.uniform(cx.min(), cx.max()), rng.uniform(0.5, 0.5 * depth.max())
        m = (np.abs(cx - x0) <= rng.uniform(1, 8)) & (np.abs(depth - z0) <= rng.uniform(0.5, 4))
        rho[m] = math.exp(rng.uniform(math.log(10), math.log(1000)))
        pha[m] = -rng.uniform(1, 30)
    return synth.sigma_from(rho, pha)


def geometric_factors(mesh, enr, strnr, vnr):
    x, y = mesh.node_xy(enr)
    a, b, m, n = strnr % 10000 - 1, strnr // 10000 - 1, vnr % 10000 - 1, vnr // 10000 - 1

    def inv(i, j):
        return 1.0 / np.hypot(x[i] - x[j], y[i] - y[j])

    return 2 * math.pi / ((inv(b, n) - inv(a, n)) - (inv(b, m) - inv(a, m)))


def noisy(response, rng):
    """Data and weights from a response -ln V: 3 % of magnitude, 0.1 mrad of phase."""
    mag = np.exp(-response.real) * (1.0 + 0.03 * rng.standard_normal(len(response)))
    pha = -response.imag + 1e-4 * rng.standard_normal(len(response))
    return -np.log(np.abs(mag)) - 1j * pha, np.full(len(response), 1.0 / 0.03 ** 2)


def kernel_jacobian(mesh, enr, strnr, vnr, rng):
    """Sensitivities as a program of its own would hold them: line sources over a half-space at the cells'
    centres, each reading's row summing to one, with the cells' phases."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    cx, cy = (torch.tensor(v, device=dev) for v in synth.centroids(mesh))
    nodes = np.asarray(mesh.nrel[: mesh.elanz, : int(mesh.selanz[0])])
    px, py = mesh.node_xy(nodes)
    area = torch.tensor(0.5 * np.abs((px * np.roll(py, -1, 1) - py * np.roll(px, -1, 1)).sum(1)), device=dev)
    x, y = (torch.tensor(v, device=dev) for v in mesh.node_xy(enr))
    dx, dy = cx[:, None] - x[None, :], cy[:, None] - y[None, :]
    r2 = dx * dx + dy * dy + 0.01
    gx, gy = dx / r2, dy / r2
    a, b, m, n = (torch.tensor(v.astype(np.int64) - 1, device=dev)
                  for v in (strnr % 10000, strnr // 10000, vnr % 10000, vnr // 10000))
    J = area[:, None] * ((gx[:, a] - gx[:, b]) * (gx[:, m] - gx[:, n]) + (gy[:, a] - gy[:, b]) * (gy[:, m] - gy[:, n]))
    J = J / J.sum(0, keepdim=True).abs().clamp_min(1e-3 * J.abs().sum(0, keepdim=True))
    J = J.to(torch.complex128) * torch.exp(1j * torch.tensor(rng.uniform(-0.03, 0.03, mesh.elanz), device=dev))[:, None]
    J = J.cpu().numpy()          # [manz, nanz]: column j of sens(nanz, manz) is contiguous
    model = np.log(ground(mesh, rng)) - np.log(0.01)
    data = J.T @ model
    data = data + 0.03 * rng.standard_normal(len(data)) + 1e-4j * rng.standard_normal(len(data))
    return J.T, data


def batch_cases(c):
    """The uneven instances of a batch: sizes between a fifth of the case's cells and all of them."""
    out = []
    for i in range(c["count"]):
        f = 0.2 ** (((i * 5) % c["count"]) / max(1, c["count"]))
        nx = max(24, int(c["nx"] * math.sqrt(f)))
        out.append({**c, "kind": "start", "count": 1, "nx": nx, "nz": max(8, int(c["nz"] * math.sqrt(f)) + i % 3),
                    "nel": max(10, min(c["nel"], int(c["nel"] * math.sqrt(f)) + i % 5, nx - 8))})
    return out


def inputs(c, seed):
    """The numbers a case's calls take, as numpy arrays, by its seed alone."""
    mesh, enr, strnr, vnr, reg = survey(frozen(c))
    rng = np.random.default_rng([seed, 20261205])
    if c["kind"] in ("forward", "sens", "start"):
        return dict(sigma=ground(mesh, rng))
    par0 = np.full(mesh.elanz, np.log(0.01) + 0j)
    lam = c["lam"] * float(max(mesh.elanz, len(strnr)))
    if c["kind"] == "gn":
        return dict(sigma=ground(mesh, rng), rng=rng, par=par0, lam=lam)
    J, data = kernel_jacobian(mesh, enr, strnr, vnr, rng)
    lams = lam * 10.0 ** np.linspace(0.5, -1.0, c["count"])
    return dict(J=J, dat=data, wmatd=np.full(len(data), 1.0 / 0.03 ** 2), par=par0, lam=lam, lams=lams,
                response=np.zeros(len(data), np.complex128))


# -- the calls ----------------------------------------------------------------

def context(c):
    mesh, enr, strnr, vnr, reg = survey(frozen(c))
    ctx = Context(mesh, enr, strnr, vnr, precision=PREC_MIXED if c["mixed"] else PREC_FP64)
    if reg is not None:
        ctx.set_regularizer(**reg)
    return ctx


def prepare(c, seed):
    if c["kind"] == "batch":
        parts = batch_cases(c)
        ctxs = [context(p) for p in parts]
        sigmas = [inputs(p, seed + 1000 * i)["sigma"] for i, p in enumerate(parts)]
        batch = Batch(ctxs, jacobian_mode=0)
        batch.set_models(sigmas)
        batch.run()              # the program's first run builds its graph
        return dict(c=c, ctxs=ctxs, batch=batch, sigmas=sigmas)
    ctx, s = context(c), inputs(c, seed)
    mesh, enr, strnr, vnr, _ = survey(frozen(c))
    if c["kind"] == "forward" and not c["dc"]:
        s["kfak"] = geometric_factors(mesh, enr, strnr, vnr)
    if c["kind"] == "start":
        ctx.set_data(np.zeros(len(strnr), np.complex128), np.full(len(strnr), 1.0 / 0.03 ** 2))
    if c["kind"] == "gn":
        _, response = ctx.forward(s["sigma"], ldc=c["dc"])
        s["dat"], s["wmatd"] = noisy(response, s["rng"])
    if "J" in s:
        ctx.set_jacobian(s.pop("J"))
    if "dat" in s:
        ctx.set_data(s["dat"], s["wmatd"])
    if c["kind"] in ("gn", "update", "trials"):
        # the reference's stop rule and cap in its own (Jacobi) form, a relative residual of 1e-6 in the block form
        s["prm"] = Context.params(s["lam"], eps=1e-12 if c["block"] else 1e-4,
                                  ncgmax=2000 if c["block"] else max(10, mesh.elanz // 10), ldc=c["dc"],
                                  precond=PRECOND_BLOCK if c["block"] else PRECOND_JACOBI)
    return dict(c=c, ctx=ctx, **s)


def run(s):
    c = s["c"]
    if c["kind"] == "batch":
        s["batch"].set_models(s["sigmas"])
        s["batch"].run()
        return [s["batch"].results(i) + (x.coverage(weight=np.ones(x.nanz)),) for i, x in enumerate(s["ctxs"])]
    ctx = s["ctx"]
    if c["kind"] == "forward":
        volt, response = ctx.forward(s["sigma"], ldc=c["dc"], mode=0 if c["dc"] else 1, kfak=s.get("kfak"))
        return dict(volt=volt, response=response)
    if c["kind"] == "sens":
        volt, response = ctx.forward(s["sigma"], mode=1)
        return dict(volt=volt, response=response, sens=ctx.jacobian(mode=2))
    if c["kind"] == "start":
        volt, response = ctx.forward(s["sigma"], ldc=c["dc"])
        ctx.jacobian(mode=1 if c["dc"] else 0, copy=False)
        return dict(volt=volt, response=response, lam0=ctx.blam0(1.0, 1.0, ldc=c["dc"]), coverage=ctx.coverage())
    if c["kind"] == "gn":
        got = ctx.gn_step(s["prm"], s["par"])
        return dict(par=got["par"], response=got["sigmaa"])
    if c["kind"] == "update":
        got = ctx.update(s["prm"], s["par"], sigmaa=s["response"])
        return dict(par=got["par"], dpar=got["dpar"], cgfac=got["cgfac"])
    got = ctx.update_lambdas(s["prm"], s["lams"], s["par"], sigmaa=s["response"])
    return dict(par=got["par"], dpar=got["dpar"])


def work(c):
    """Band Cholesky per wavenumber and two substitutions per electrode; for the sensitivities the products
    of all electrode pairs and one write of the Jacobian; for an inner solve one read of it.  Complex
    multiply-adds are 8 flops, real ones 2."""
    if c["kind"] == "batch":
        parts = [work(p) for p in batch_cases(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    mesh, enr, strnr, vnr, _ = survey(frozen(c))
    n, E, L, N, mb = mesh.sanz, mesh.elanz, len(enr), len(strnr), mesh.mb
    mac, num = (2.0, 8) if c["dc"] else (8.0, 16)
    entry = num // 2 if c["mixed"] else num
    if c["kind"] in ("update", "trials"):
        return {"bytes": float(N * E * entry + c["count"] * 3 * num * E), "flops": 2 * mac * N * E * c["count"]}
    K = len(wavenumbers(mesh, enr, strnr, vnr)[0])
    w = {"bytes": 16.0 * E + 32.0 * N, "flops": K * mac * (0.5 * n * mb * mb + 2.0 * n * mb * L)}
    if c["kind"] != "forward":
        w["bytes"] += float(N * E * entry)
        w["flops"] += mac * E * K * L * (L + 1) / 2 * int(mesh.selanz[0]) * 2
    if c["kind"] == "gn":
        w["bytes"] += float(N * E * entry)
        w["flops"] += 2 * mac * N * E
    return w


# -- the same in plain 64-bit torch ---------------------------------------------

def wavenumbers(mesh, enr, strnr, vnr):
    """Gauss-Legendre (in sqrt k) and Gauss-Laguerre nodes by the ratio of the largest to the smallest
    distance between a current and a potential electrode."""
    x, y = mesh.node_xy(enr)
    d = [np.hypot(x[i - 1] - x[j - 1], y[i - 1] - y[j - 1])
         for i in (strnr % 10000, strnr // 10000) for j in (vnr % 10000, vnr // 10000)]
    lo, hi = min(v.min() for v in d), max(v.max() for v in d)
    ng = min(max(int(np.float32(6.0 * math.log10(hi / lo))), 2), 26)
    k0 = 1.0 / (2.0 * lo)
    t, w = np.polynomial.legendre.leggauss(ng)
    t, w = 0.5 * (t + 1.0), 0.5 * w
    u, v = np.polynomial.laguerre.laggauss(4)
    return np.concatenate([k0 * t * t, k0 * (u + 1.0)]), np.concatenate([2.0 * k0 * w * t, k0 * v * np.exp(u)])


def bessel_ratio_terms(x):
    """K0 and K1 by the polynomials of Abramowitz and Stegun 9.8.1 to 9.8.8, zero beyond 500."""
    def poly(t, a):
        return np.polynomial.polynomial.polyval(t, a)

    with np.errstate(all="ignore"):
        t = (x / 3.75) ** 2
        i0 = poly(t, [1.0, 3.5156229, 3.0899424, 1.2067492, 0.2659732, 0.0360768, 0.0045813])
        i1 = x * poly(t, [0.5, 0.87890594, 0.51498869, 0.15084934, 0.02658733, 0.00301532, 0.00032411])
        q = x * x / 4.0
        k0s = -np.log(x / 2.0) * i0 + poly(q, [-0.57721566, 0.42278420, 0.23069756, 0.03488590, 0.00262698, 0.00010750,
                                              0.0000074])
        k1s = np.log(x / 2.0) * i1 + poly(q, [1.0, 0.15443144, -0.67278579, -0.18156897, -0.01919402, -0.00110404,
                                             -0.00004686]) / x
        z = 2.0 / x
        f = np.exp(-x) / np.sqrt(x)
        k0l = f * poly(z, [1.25331414, -0.07832358, 0.02189568, -0.01062446, 0.00587872, -0.00251540, 0.00053208])
        k1l = f * poly(z, [1.25331414, 0.23498619, -0.03655620, 0.01504268, -0.00780353, 0.00325614, -0.00068245])
    return (np.where(x <= 2.0, k0s, np.where(x > 500.0, 0.0, k0l)),
            np.where(x <= 2.0, k1s, np.where(x > 500.0, 0.0, k1l)))


def triangle(x, y):
    """Stiffness and mass matrices of linear triangles (counter-clockwise nodes in the last axis)."""
    bx = np.roll(y, -1, -1) - np.roll(y, -2, -1)
    by = np.roll(x, -2, -1) - np.roll(x, -1, -1)
    det = (x[..., 1] - x[..., 0]) * (y[..., 2] - y[..., 0]) - (x[..., 2] - x[..., 0]) * (y[..., 1] - y[..., 0])
    det = det[..., None, None]
    stiff = (bx[..., :, None] * bx[..., None, :] + by[..., :, None] * by[..., None, :]) / (2.0 * det)
    return stiff, det * (np.ones((3, 3)) + np.eye(3)) / 24.0


def cell_matrices(mesh, k):
    """[E, nodes, nodes] at wavenumber k; a quadrilateral is four triangles around the crossing of its
    diagonals, that node condensed out."""
    nodes = np.asarray(mesh.nrel[: mesh.elanz, : int(mesh.selanz[0])])
    x, y = mesh.node_xy(nodes)
    if nodes.shape[1] == 3:
        stiff, mass = triangle(x, y)
        return stiff + k * k * mass
    a, b = (y[:, 2] - y[:, 0]) / (x[:, 2] - x[:, 0]), (y[:, 3] - y[:, 1]) / (x[:, 3] - x[:, 1])
    xc = (a * x[:, 0] - y[:, 0] - b * x[:, 1] + y[:, 1]) / (a - b)
    x5 = np.column_stack([x, xc])
    y5 = np.column_stack([y, y[:, 0] + a * (xc - x[:, 0])])
    full = np.zeros((len(x), 5, 5))
    for t in ([0, 1, 4], [1, 2, 4], [4, 2, 3], [0, 4, 3]):
        stiff, mass = triangle(x5[:, t], y5[:, t])
        full[np.ix_(range(len(x)), t, t)] += stiff + k * k * mass
    return full[:, :4, :4] - full[:, :4, 4:] * full[:, 4:, :4] / full[:, 4:, 4:]


def potentials(c, sigma, k):
    """[nodes, electrodes]: the potentials of unit sources at wavenumber k, and the cells' matrices."""
    mesh, enr, _, _, _ = survey(frozen(c))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n, E, L = mesh.sanz, mesh.elanz, len(enr)
    dt = torch.float64 if c["dc"] else torch.complex128
    sig = torch.tensor(sigma.real if c["dc"] else sigma, device=dev, dtype=dt)
    cells = torch.tensor(cell_matrices(mesh, k), device=dev)
    nodes = torch.tensor(np.asarray(mesh.nrel[:E, : cells.shape[1]], np.int64) - 1, device=dev)
    A = torch.zeros(n * n, device=dev, dtype=dt)
    A.index_add_(0, (nodes[:, :, None] * n + nodes[:, None, :]).reshape(-1), (cells * sig[:, None, None]).reshape(-1))
    A = A.reshape(n, n)
    src = torch.tensor(enr.astype(np.int64) - 1, device=dev)
    rhs = torch.zeros(n, L, device=dev, dtype=dt)
    rhs[src, torch.arange(L, device=dev)] = 1.0
    r11 = int(mesh.nelanz[1])          # the surface segments come first, then the sides and the bottom
    side = np.asarray(mesh.nrel[E + r11:, :2], np.int64) - 1
    inside = torch.ones(n, dtype=torch.bool, device=dev)
    inside[torch.tensor(np.unique(side), device=dev)] = False
    I, G = torch.nonzero(inside)[:, 0], torch.nonzero(~inside)[:, 0]
    out = torch.zeros(n, L, device=dev, dtype=dt)
    if c["dirichlet"]:
        out[I] = torch.linalg.solve(A[I][:, I], rhs[I])
        return out, cells, nodes, sig
    m = len(G)
    AIG = A[I][:, G]
    X = torch.linalg.solve(A[I][:, I], torch.cat([AIG, rhs[I]], 1))
    S0, g0 = A[G][:, G] - AIG.T @ X[:, :m], rhs[G] - AIG.T @ X[:, m:]
    # the sides' condition, a function of the source: k (cos K1 + cos' K1') / (K0 + K0') with the mirrored source
    px, py = mesh.node_xy(side + 1)
    ex, ey = mesh.node_xy(enr)
    xr, yr = px.mean(1)[:, None], py.mean(1)[:, None]
    tx, ty = (py[:, 0] - py[:, 1])[:, None], (px[:, 1] - px[:, 0])[:, None]
    length = np.hypot(tx, ty)
    terms = []
    for dy in (yr - ey[None, :], yr + ey[None, :]):
        dx = xr - ex[None, :]
        r = np.hypot(dx, dy)
        terms.append(((dx * tx + dy * ty) / r / length, *bessel_ratio_terms(r * k)))
    (cm, k0m, k1m), (cp, k0p, k1p) = terms
    with np.errstate(all="ignore"):
        beta = k * np.where(k0m + k0p == 0.0, (cm + cp) / 2.0, (cm * k1m + cp * k1p) / (k0m + k0p))
    pos = torch.zeros(n, dtype=torch.long, device=dev)
    pos[G] = torch.arange(m, device=dev)
    sg = pos[torch.tensor(side, device=dev)]
    rnr = torch.tensor(np.asarray(mesh.rnr[r11:], np.int64) - 1, device=dev)
    coef = torch.tensor(beta * length / 6.0, device=dev) * sig[rnr][:, None]      # [segments, electrodes]
    S = S0.expand(L, m, m).reshape(L, m * m).clone()
    for i in range(2):
        for j in range(2):
            S.index_add_(1, sg[:, i] * m + sg[:, j], (coef * (2.0 if i == j else 1.0)).T.contiguous())
    pg = torch.linalg.solve(S.reshape(L, m, m), g0.T[:, :, None])[:, :, 0].T
    out[G] = pg
    out[I] = X[:, m:] - X[:, :m] @ pg
    return out, cells, nodes, sig


def exact_forward(c, sigma, want_sens):
    """Voltages, and sens [manz, nanz] without the factor sigma / V."""
    mesh, enr, strnr, vnr, _ = survey(frozen(c))
    kw, wt = wavenumbers(mesh, enr, strnr, vnr)
    a, b, m, n = strnr % 10000 - 1, strnr // 10000 - 1, vnr % 10000 - 1, vnr // 10000 - 1
    volt, sens = 0.0, 0.0
    for k, w in zip(kw, wt):
        phi, cells, nodes, sig = potentials(c, sigma, k)
        el = phi[torch.tensor(enr.astype(np.int64) - 1, device=phi.device)] * (w / math.pi)
        volt = volt + ((el[n, b] - el[n, a]) - (el[m, b] - el[m, a]))
        if want_sens:
            ds, dp = phi[:, b] - phi[:, a], phi[:, n] - phi[:, m]
            for i in range(nodes.shape[1]):
                t = sum(cells[:, i, j][:, None] * ds[nodes[:, j]] for j in range(nodes.shape[1]))
                sens = sens + t * dp[nodes[:, i]] * (w / math.pi)
    return volt, sens, sig


def regulariser(reg, M):
    """The smoothness operator as a dense matrix."""
    sm = torch.tensor(np.ascontiguousarray(reg["smatm"]))
    R = torch.zeros(M, M, dtype=torch.float64)
    i = torch.arange(M)
    if reg["ltri"] == 0:
        nx = reg["nx"]
        R[i, i] = sm[:, 0]
        R[i[:-1], i[1:]] = sm[:-1, 1]
        R[i[1:], i[:-1]] = sm[:-1, 1]
        R[i[:-nx], i[nx:]] = sm[:-nx, 2]
        R[i[nx:], i[:-nx]] = sm[:-nx, 2]
        return R
    nb = torch.tensor(np.ascontiguousarray(reg["nachbar"]).astype(np.int64))
    for q in range(nb.shape[1] - 1):
        has = nb[:, q] > 0
        R[i[has], nb[has, q] - 1] = sm[has, q]
    R[i, i] = sm[:, -1]
    return R


def exact_update(J, R, wd, resid, par, lam, prm):
    """par + the update: the solution of the normal equations in the block form, the reference's truncated
    conjugate gradients otherwise.  J is [manz, nanz] (real or complex)."""
    g = J.conj() @ (wd * resid) - lam * (R @ par)
    fac = 1.0 / torch.sqrt((J.abs() ** 2) @ wd.real + lam * R.diagonal().real)
    if prm.precond == PRECOND_BLOCK:
        H = (J.conj() * wd) @ J.T + lam * R
        d = torch.cholesky_solve(g[:, None], torch.linalg.cholesky(H))[:, 0]
        return par + d, d, fac
    r = g * fac
    x, p, dr1, dr0 = torch.zeros_like(r), torch.zeros_like(r), 0.0, 0.0
    for it in range(prm.ncgmax):
        dr = float(torch.vdot(r, r).real)
        if it == 0:
            dr0 = dr * prm.eps
        elif dr <= dr0:
            break
        p = r + (dr / dr1 if it else 0.0) * p
        q = fac * (J.conj() @ (wd * (J.T @ (fac * p))) + lam * (R @ (fac * p)))
        alpha = dr / float(torch.vdot(p, q).real)
        x, r, dr1 = x + alpha * p, r - alpha * q, dr
    d = x * fac
    return par + d, d, fac


def exact(c, seed):
    if c["kind"] == "batch":
        got = [exact(p, seed + 1000 * i) for i, p in enumerate(batch_cases(c))]
        return [(g["volt"], g["response"], g["unit_coverage"]) for g in got]
    mesh, enr, strnr, vnr, reg = survey(frozen(c))
    if mesh.sanz > 21000 or (c["kind"] in ("gn", "update", "trials") and mesh.elanz > 10000):
        return None
    s = inputs(c, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if c["kind"] in ("update", "trials"):
        J = torch.tensor(s["J"].T, device=dev)
        R = regulariser(reg, mesh.elanz).to(dev).to(J.dtype)
        wd, dat, par = (torch.tensor(s[k], device=dev).to(J.dtype) for k in ("wmatd", "dat", "par"))
        lams = s["lams"] if c["kind"] == "trials" else [s["lam"]]
        prm = Context.params(0.0, eps=1e-4, ncgmax=max(10, mesh.elanz // 10))
        J2 = J.abs() ** 2
        got = []
        for lam in lams:
            x, d, _ = exact_update(J, R, wd, dat, par, float(lam), prm)
            got.append((x, d))
        if c["kind"] == "trials":
            return dict(par=torch.stack([g[0] for g in got]), dpar=torch.stack([g[1] for g in got]))
        fac = 1.0 / torch.sqrt(J2 @ wd.real + s["lam"] * R.diagonal().real)
        return dict(par=got[0][0], dpar=got[0][1], cgfac=fac)
    if c["kind"] != "gn":
        volt, sens, sig = exact_forward(c, s["sigma"], c["kind"] != "forward")
        cvolt = volt.to(torch.complex128)
        if c["kind"] == "forward" and not c["dc"]:
            kfak = torch.tensor(geometric_factors(mesh, enr, strnr, vnr), device=dev)
            return dict(volt=cvolt, response=kfak * cvolt)
        if c["kind"] == "sens":
            return dict(volt=cvolt, response=cvolt, sens=-sens.T)
        if c["kind"] == "forward":
            return dict(volt=cvolt, response=-torch.log(cvolt))
        J = sens * (sig[:, None] / volt[None, :])
        w = 1.0 / 0.03 ** 2
        s1 = J.sum(0) * w
        lam0 = float(5.0 * (J.conj() @ s1).abs().sum() / mesh.elanz)
        return dict(volt=cvolt, response=-torch.log(cvolt), lam0=lam0, coverage=J.abs().sum(1) * math.sqrt(w),
                    unit_coverage=J.abs().sum(1))
    volt, _, _ = exact_forward(c, s["sigma"], False)
    dat, wmatd = noisy(-np.log(volt.to(torch.complex128).cpu().numpy()), s["rng"])
    volt, sens, sig = exact_forward(c, np.exp(s["par"]), True)
    J = sens * (sig[:, None] / volt[None, :])
    R = regulariser(reg, mesh.elanz).to(dev).to(J.dtype)
    response = -torch.log(volt.to(torch.complex128))
    pick = (lambda v: v.real) if c["dc"] else (lambda v: v)
    prm = Context.params(s["lam"], eps=1e-4, ncgmax=max(10, mesh.elanz // 10),
                         precond=PRECOND_BLOCK if c["block"] else PRECOND_JACOBI)
    par = torch.tensor(s["par"], device=dev)
    _, d, _ = exact_update(J, R, torch.tensor(wmatd, device=dev).to(J.dtype),
                           pick(torch.tensor(dat, device=dev) - response), pick(par), s["lam"], prm)
    return dict(par=par + d, response=response)
