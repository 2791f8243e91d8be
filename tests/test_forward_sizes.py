"""Forward potentials at the sizes where the kernels' tiles,
panels and row blocks have remainders, against the oracle."""
import numpy as np
import pytest

from crtomo_stable_b200 import synth

RTOL = 1e-10       # of the largest potential / voltage: the other parity tests' bound


def survey(nx, nz, nel, tri, seed=3):
    rng = np.random.default_rng(seed)
    xs = np.arange(nx + 1, dtype=np.float64) - (nx - nel) // 2
    mesh = synth.structured_mesh(xs, synth.graded_depths(nz, 0.4, 1.0 + 2.0 / nz), triangles=tri)
    enr = synth.surface_electrodes(mesh, xs, np.arange(nel, dtype=np.float64), nz)
    configs = synth.dipole_dipole(nel, (1, 2), 6) if nel >= 4 else [(1, 0, 2, 0)]
    strnr, vnr = synth.encode(configs)
    rho = np.exp(rng.uniform(np.log(10.0), np.log(1000.0), mesh.elanz))
    return mesh, enr, strnr, vnr, synth.sigma_from(rho, -rng.uniform(1.0, 30.0, mesh.elanz))


# (cells, cells, electrodes, triangles): half-bandwidths 4 to 131, boundary
# sets of 9 to 350 nodes, interiors of a single panel up to 6,400 rows
SIZES = [(4, 2, 2, True), (6, 3, 4, False), (9, 7, 5, True), (33, 8, 17, False), (20, 31, 12, True),
         (40, 15, 33, True), (24, 64, 10, False), (20, 80, 9, True), (16, 127, 7, True), (28, 130, 9, True),
         (180, 36, 96, True)]


@pytest.mark.gpu
@pytest.mark.parametrize("ldc", [False, True])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(str(int(v)) for v in s))
def test_forward_potentials(size, ldc):
    from crtomo_stable_b200.lib import FORWARD_SCHUR, Context
    from oracle.oracle import OracleProblem
    mesh, enr, strnr, vnr, sigma = survey(*size)
    ctx = Context(mesh, enr, strnr, vnr)
    op = OracleProblem(mesh, enr, strnr, vnr, kwn=ctx.kwn, kwnwi=ctx.kwnwi)
    kp_o = op.forward(sigma, ldc=ldc, nthreads=8)
    volt_o, _ = op.bvolti(op.rtrafo(kp_o))
    volt, _, kp = ctx.forward(sigma, ldc=ldc, want_kpot=True)
    assert ctx.forward_info()[0] == FORWARD_SCHUR
    assert np.abs(kp - kp_o).max() <= RTOL * np.abs(kp_o).max()
    assert np.abs(volt - volt_o).max() <= RTOL * np.abs(volt_o).max()
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz,panel", [(12, 2, 4), (14, 7, 4), (14, 16, 4), (15, 17, 4), (14, 25, 4), (14, 33, 4),
                                         (13, 41, 4), (13, 57, 4), (12, 66, 4), (12, 75, 4), (12, 77, 8), (12, 88, 8),
                                         (12, 90, 4), (12, 100, 4), (12, 106, 8), (12, 112, 8), (12, 127, 8)])
def test_factor_in_registers_is_the_panel_blocked_factor(nx, nz, panel, monkeypatch):
    """The interior factor with its window in registers against the
    panel-blocked kernel at the panel width whose order of products it keeps:
    the same potentials bit for bit, complex and real."""
    from crtomo_stable_b200.lib import Context
    mesh, enr, strnr, vnr, sigma = survey(nx, nz, 5, nz % 2 == 0)
    out = []
    for blocked in (False, True):
        if blocked:
            monkeypatch.setenv("CRT_B200_PANEL", str(panel))
        ctx = Context(mesh, enr, strnr, vnr)
        out.append([ctx.forward(sigma, ldc=ldc, want_kpot=True)[2] for ldc in (False, True)])
        ctx.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("solve", ["direct", "iter"])
@pytest.mark.parametrize("ldc", [False, True])
@pytest.mark.parametrize("nx,nz,nel", [(5, 2, 2), (12, 5, 9), (30, 12, 17), (80, 40, 6), (150, 90, 5), (380, 80, 3)])
def test_boundary_systems(nx, nz, nel, ldc, solve, monkeypatch):
    """The electrodes' boundary systems (9 to 541 nodes: the factor in shared
    memory, staged, and above the staged form's 536 complex nodes) by their
    Cholesky factors and by the preconditioned iteration, against the oracle."""
    from crtomo_stable_b200.lib import FORWARD_SCHUR, Context
    from oracle.oracle import OracleProblem
    mesh, enr, strnr, vnr, sigma = survey(nx, nz, nel, False)
    kwn, kwnwi = np.array([0.02, 0.3]), np.array([0.1, 0.2])
    monkeypatch.setenv("CRT_B200_SCHUR_SOLVE", solve)
    ctx = Context(mesh, enr, strnr, vnr, kwn=kwn, kwnwi=kwnwi)
    kp = ctx.forward(sigma, ldc=ldc, want_kpot=True)[2]
    assert ctx.forward_info()[0] == FORWARD_SCHUR
    kp_o = OracleProblem(mesh, enr, strnr, vnr, kwn=kwn, kwnwi=kwnwi).forward(sigma, ldc=ldc, nthreads=8)
    assert np.abs(kp - kp_o).max() <= RTOL * np.abs(kp_o).max()
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz,nel", [(4, 2, 2), (9, 6, 4), (20, 7, 12), (18, 15, 9), (23, 16, 11), (40, 24, 17),
                                       (30, 64, 9), (16, 121, 7), (16, 127, 7)])
def test_sweeps_paired_or_alone(nx, nz, nel, monkeypatch):
    """The triangular sweeps with two CTAs on an SM (launches of more CTAs
    than SMs) and with one: a wavenumber's potentials are the same bit for bit
    in a launch of 160 and alone, complex and real."""
    from crtomo_stable_b200.lib import FORWARD_SCHUR, Context
    monkeypatch.setenv("CRT_B200_SCHUR_SOLVE", "direct")
    mesh, enr, strnr, vnr, sigma = survey(nx, nz, nel, True)
    kwn = np.geomspace(0.01, 2.0, 160)
    many = Context(mesh, enr, strnr, vnr, kwn=kwn, kwnwi=np.ones(160))
    one = Context(mesh, enr, strnr, vnr, kwn=kwn[77:78], kwnwi=np.ones(1))
    for ldc in (False, True):
        a = many.forward(sigma, ldc=ldc, want_kpot=True)[2]
        assert many.forward_info()[0] == FORWARD_SCHUR
        b = one.forward(sigma, ldc=ldc, want_kpot=True)[2]
        assert np.array_equal(a[..., 77], b[..., 0])
    many.close()
    one.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz,nel,tri", [(9, 3, 4, False), (14, 4, 8, True), (15, 4, 9, False), (24, 4, 16, True),
                                           (25, 4, 17, False), (40, 3, 33, True), (55, 3, 48, False), (70, 3, 64, True),
                                           (71, 3, 65, False), (120, 3, 113, True), (134, 3, 128, True),
                                           (135, 3, 129, False)])
def test_sensitivities_gram_against_direct(nx, nz, nel, tri, monkeypatch):
    """The Gram form of the sensitivities at electrode counts where its tiles
    and units have remainders (129: above the tensor form) against the
    per-reading form.  A sum of 200 products rounds to 2e-14 of the largest;
    the four-term combination leaves at least 1e-4 of it at a reading's
    largest sensitivity, hence 1e-9 of that."""
    from crtomo_stable_b200.lib import Context
    mesh, enr, strnr, vnr, sigma = survey(nx, nz, nel, tri)
    for mode in (0, 1, 2):
        out = []
        for kern in ("gram", "direct"):
            if kern == "direct":
                monkeypatch.setenv("CRT_B200_SENS", "direct")
            else:
                monkeypatch.delenv("CRT_B200_SENS", raising=False)
            ctx = Context(mesh, enr, strnr, vnr)
            ctx.forward(sigma, ldc=mode == 1)
            out.append(ctx.jacobian(mode=mode))
            ctx.close()
        assert (np.abs(out[0] - out[1]) <= 1e-9 * np.abs(out[1]).max(axis=1, keepdims=True)).all()


@pytest.mark.gpu
@pytest.mark.parametrize("nz,tri", [(z, z % 2 == 1) for z in range(1, 19)])
def test_sweeps_in_narrow_bands(nz, tri):
    """Interior half-bandwidths of 1 to 18, below and above the sweeps'
    blocks of 16 rows, over many blocks, two streams at once: the potentials
    of the per-electrode band form, and the same bits from run to run."""
    from concurrent.futures import ThreadPoolExecutor

    from crtomo_stable_b200.lib import FORWARD_DIRECT, FORWARD_SCHUR, Context
    mesh, enr, strnr, vnr, sigma = survey(150, nz, 12, tri)
    kwn = np.geomspace(0.01, 2.0, 24)
    ctxs = [Context(mesh, enr, strnr, vnr, kwn=kwn, kwnwi=np.ones(24)) for _ in range(2)]
    for ldc in (False, True):
        def runs(ctx):
            return [ctx.forward(sigma, ldc=ldc, want_kpot=True)[2] for _ in range(4)]
        for c in ctxs:
            c.set_forward_form(FORWARD_SCHUR)
        with ThreadPoolExecutor(2) as ex:
            first, *more = [kp for out in ex.map(runs, ctxs) for kp in out]
        assert all(np.array_equal(first, kp) for kp in more)
        ctxs[0].set_forward_form(FORWARD_DIRECT)
        ref = runs(ctxs[0])[0]
        assert np.abs(first - ref).max() <= RTOL * np.abs(ref).max()
    for c in ctxs:
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("col", [1, 2, 3, 17, 30, 44, 57, 58])
def test_pivot_breakdown_in_registers(col):
    """A negative cell makes the interior system indefinite at its column of
    the mesh (early, middle and last panels of the factor): an error, and the
    next forward on the context gives the bits of the one before."""
    from crtomo_stable_b200.lib import CRTError, FORWARD_SCHUR, Context
    mesh, enr, strnr, vnr, _ = survey(60, 20, 9, False)
    sigma = np.full(mesh.elanz, 0.01, np.complex128)
    ctx = Context(mesh, enr, strnr, vnr)
    kp = ctx.forward(sigma, ldc=True, want_kpot=True)[2]
    assert ctx.forward_info()[0] == FORWARD_SCHUR
    bad = sigma.copy()
    bad[8 * 60 + col] = -0.02
    for _ in range(3):
        with pytest.raises(CRTError):
            ctx.forward(bad, ldc=True)
        assert np.array_equal(ctx.forward(sigma, ldc=True, want_kpot=True)[2], kp)
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("col", [1, 30, 57])
def test_factor_error_is_reported(col):
    """A pivot that breaks down is error 28, whether or not the sweep beside
    the factor notices first."""
    from crtomo_stable_b200.lib import CRTError, Context
    mesh, enr, strnr, vnr, _ = survey(60, 20, 9, False)
    sigma = np.full(mesh.elanz, 0.01, np.complex128)
    sigma[8 * 60 + col] = -0.02
    ctx = Context(mesh, enr, strnr, vnr)
    for _ in range(5):
        with pytest.raises(CRTError) as ei:
            ctx.forward(sigma, ldc=True)
        assert ei.value.errnr == 28
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("solve", ["direct", "iter"])
@pytest.mark.parametrize("nodes", [255, 256, 257, 399, 401, 488, 489, 527, 529, 641, 767])
def test_boundary_systems_of_many_or_few(nodes, solve, monkeypatch):
    """The boundary systems (or reference factors) of 160 wavenumbers, more
    than SMs, and of one wavenumber, at both sides of where the left-looking
    factor takes over from the right-looking one: the same bits."""
    from crtomo_stable_b200.lib import FORWARD_SCHUR, Context
    monkeypatch.setenv("CRT_B200_SCHUR_SOLVE", solve)
    mesh, enr, strnr, vnr, sigma = survey(nodes - 17, 8, 2, False)
    kwn = np.geomspace(0.01, 2.0, 160)
    many = Context(mesh, enr, strnr, vnr, kwn=kwn, kwnwi=np.ones(160))
    one = Context(mesh, enr, strnr, vnr, kwn=kwn[77:78], kwnwi=np.ones(1))
    for ldc in (False, True):
        a = many.forward(sigma, ldc=ldc, want_kpot=True)[2]
        assert many.forward_info()[:2] == (FORWARD_SCHUR, nodes)
        b = one.forward(sigma, ldc=ldc, want_kpot=True)[2]
        assert np.array_equal(a[..., 77], b[..., 0])
    many.close()
    one.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz,nel,tri", [(149, 8, 8, False), (148, 8, 8, False), (80, 8, 9, True), (80, 8, 16, True),
                                           (80, 8, 17, True), (110, 3, 72, True), (110, 3, 73, False),
                                           (110, 3, 80, True), (110, 3, 81, False), (110, 3, 96, True),
                                           (110, 3, 97, False)])
def test_sensitivities_where_the_gram_form_changes(nx, nz, nel, tri, monkeypatch):
    """Electrode and element counts at both sides of where the Gram form takes
    another kernel or another number of units per warp, as in
    test_sensitivities_gram_against_direct."""
    test_sensitivities_gram_against_direct(nx, nz, nel, tri, monkeypatch)
