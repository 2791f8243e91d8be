"""The Jacobi-form CG at the sizes where its sums over the cells have
remainders (VEC_NT = 1024 threads per sum, four elements in flight), against
the oracle: the single update, the lambda candidates, and lambda_0."""
import numpy as np
import pytest

from crtomo_stable_b200 import regularization, synth

# 12 iterations: sums of up to 4,104 terms round to about 1e-14, and a dozen
# steps carry that to 1e-12 at most
RTOL = 1e-10


@pytest.mark.gpu
@pytest.mark.parametrize("ldc", [False, True])
@pytest.mark.parametrize("nx,nz,nel", [(10, 2, 4), (31, 33, 8), (32, 32, 8), (41, 25, 9), (64, 64, 30), (72, 57, 6)])
def test_update_and_lambda_candidates(nx, nz, nel, ldc):
    from crtomo_stable_b200.lib import Context
    from oracle.oracle import OracleCG
    rng = np.random.default_rng(nx * nz)
    xs = np.arange(nx + 1, dtype=np.float64) - (nx - nel) // 2
    mesh = synth.structured_mesh(xs, synth.graded_depths(nz, 0.4, 1.01), triangles=False)
    strnr, vnr = synth.encode(synth.dipole_dipole(nel, (1, 2), 8))
    M, N = mesh.elanz, len(strnr)
    ctx = Context(mesh, synth.surface_electrodes(mesh, xs, np.arange(nel, dtype=np.float64), nz), strnr, vnr)
    sm = regularization.smatm_reg(mesh, nx, nz, 1.0, 1.0)
    J = rng.standard_normal((N, M)) if ldc else rng.standard_normal((N, M)) + 1j * rng.standard_normal((N, M))
    wd = rng.uniform(0.5, 2.0, N)
    dat = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    par = rng.standard_normal(M) + 1j * rng.standard_normal(M)
    response = np.zeros(N, np.complex128)
    ctx.set_regularizer(0, sm, nx=nx)
    ctx.set_data(dat, wd)
    ctx.set_jacobian(J, real=ldc)
    lams = [30.0 * M, 100.0 * M, 300.0 * M]
    many = ctx.update_lambdas(Context.params(0.0, eps=0.0, ncgmax=12, ldc=ldc), lams, par, sigmaa=response)
    for i, lam in enumerate(lams):
        one = ctx.update(Context.params(lam, eps=0.0, ncgmax=12, ldc=ldc), par, sigmaa=response)
        assert one["ncg"] == many["ncg"][i] == 12
        assert np.abs(one["dpar"] - many["dpar"][i]).max() <= RTOL * np.abs(one["dpar"]).max()
        cg = OracleCG(M, N, 0, sm, nx=nx, wmatd=wd, lam=lam, eps=0.0, ncgmax=12, ldc=ldc)
        ref = cg.update(None if ldc else J, dat, response, par, 1.0, sensdc=J if ldc else None)
        assert np.abs(one["dpar"] - ref["dpar"]).max() <= RTOL * np.abs(ref["dpar"]).max()
    lam0 = float(5.0 * np.abs(J.conj().T @ (wd * J.sum(1))).sum() / M)
    assert abs(ctx.blam0(1.0, 1.0, ldc=ldc) - lam0) <= 1e-12 * lam0
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz", [(192, 128), (220, 112)])
def test_update_where_the_turns_end(nx, nz):
    """24,576 cells, the most that one cluster turns an iteration over for, and
    24,640, by the grid-wide kernels."""
    test_update_and_lambda_candidates(nx, nz, 6, False)


@pytest.mark.gpu
@pytest.mark.parametrize("ldc", [False, True])
@pytest.mark.parametrize("nx,nz,nel,spacings,nmax", [(10, 2, 4, (1,), 1), (41, 25, 9, (1, 2), 8), (64, 3, 60, (1, 2), 50)])
def test_sums_of_a_formed_and_of_a_set_jacobian(nx, nz, nel, spacings, nmax, ldc):
    """lambda_0 and the coverage, whose sums lie in the Jacobian's workspace
    where it is long enough: the same from the Jacobian that the context formed
    and from the same one set on a context without that workspace, and the
    Jacobian formed again afterwards is unchanged."""
    from crtomo_stable_b200.lib import Context
    rng = np.random.default_rng(nx)
    xs = np.arange(nx + 1, dtype=np.float64) - (nx - nel) // 2
    mesh = synth.structured_mesh(xs, synth.graded_depths(nz, 0.4, 1.1), triangles=True)
    enr = synth.surface_electrodes(mesh, xs, np.arange(nel, dtype=np.float64), nz)
    strnr, vnr = synth.encode(synth.dipole_dipole(nel, spacings, nmax))
    sigma = synth.sigma_from(rng.uniform(10.0, 1000.0, mesh.elanz), -rng.uniform(1.0, 30.0, mesh.elanz))
    N = len(strnr)
    dat, wd, weight = rng.standard_normal(N) + 0j, rng.uniform(0.5, 2.0, N), rng.uniform(0.5, 2.0, N)
    kw = dict(kwn=np.array([0.05, 0.5]), kwnwi=np.array([0.1, 0.2]))
    formed, held = Context(mesh, enr, strnr, vnr, **kw), Context(mesh, enr, strnr, vnr, **kw)
    formed.forward(sigma, ldc=ldc)
    J = formed.jacobian(mode=1 if ldc else 0)
    held.set_jacobian(J, real=ldc)
    out = []
    for ctx in (formed, held):
        ctx.set_data(dat, wd)
        out.append([ctx.blam0(1.0, 1.0, ldc=ldc), ctx.coverage(), ctx.coverage(weight=weight), ctx.blam0(1.0, 1.0, ldc=ldc)])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert out[0][0] == out[0][3]
    assert np.array_equal(formed.jacobian(mode=1 if ldc else 0), J)
    formed.close()
    held.close()
