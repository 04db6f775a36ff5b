"""GPU-vs-oracle parity of the solver building blocks, called through the C ABI.

Sizes are chosen so the FP64 oracle finishes in seconds.  Tolerances: the
native path computes the same FP64 arithmetic in a different summation order
(node-centric gathers instead of accumarray scatters, a nested-dissection
factorisation instead of a permuted sparse Cholesky), so single operators agree
to ~1e-13 relative and iterative solves to ~1e-9.
"""
import numpy as np
import pytest

from oracle import top3dxl_oracle as O

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(np.ravel(a) - np.ravel(b)) / max(np.linalg.norm(np.ravel(b)), 1e-300))


@pytest.fixture(scope="module", params=["cuboid", "irregular", "u_shape"])
def setup(request):
    # u_shape: most (x, z) columns are void, so the level-1 passes run over the domain's tiles
    # and chunks only: K*u tiles with part of their z-chunk present, the last-row kernel's row
    # tiles (ny = 32), the filter's tiles, the restriction's column mask
    from top3d_xl_b200 import Context
    if request.param == "cuboid":
        vox = np.ones((12, 24, 12), bool)
    elif request.param == "u_shape":
        vox = np.zeros((32, 64, 32), bool)
        vox[:, :4, :] = True
        vox[:, -4:, :] = True
        vox[:, :, :4] = True
    else:
        rng = np.random.default_rng(5)
        vox = rng.random((13, 27, 11)) < 0.75
        vox[:, 0, :] = True
        vox[:, -1, :] = True
    m = O.build_model(vox)
    ctx = Context("fp64")
    ctx.load_voxels(vox)
    rng = np.random.default_rng(1)
    x = rng.uniform(0.05, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    ctx.set_moduli(E)
    ctx.assemble()
    yield dict(m=m, ctx=ctx, sol=sol, E=E, x=x, vox=vox, kind=request.param)
    ctx.close()


def test_ku(setup):
    m, ctx, sol = setup["m"], setup["ctx"], setup["sol"]
    u = np.random.default_rng(2).standard_normal(m.levels[0].numDOFs)
    y = ctx.ku(u)
    assert _rel(y, sol.ku(u)) < 1e-13


def test_diagonals(setup):
    m, ctx = setup["m"], setup["ctx"]
    for l in range(1, m.numLevels):
        assert _rel(ctx.diag(l), m.levels[l - 1].diagK) < 1e-13, l


def test_vcycle(setup):
    m, ctx, sol = setup["m"], setup["ctx"], setup["sol"]
    r = np.random.default_rng(3).standard_normal(m.levels[0].numDOFs)
    # the U's prongs are cantilevers: its coarsest matrix is ill-conditioned (the V-cycle of a unit
    # residual reaches 1e4), and the two factorisations' rounding differs by that much more
    bar = 1e-10 if setup["kind"] == "u_shape" else 1e-11
    assert _rel(ctx.vcycle(r), sol.vcycle(r)) < bar


def test_pcg(setup):
    # the tol-1e-3 PCG amplifies rounding ~1e8 (tests/test_oracle.py): on this
    # high-contrast random design the solution agrees to ~1e-8 and f'u to ~1e-9
    m, ctx, sol = setup["m"], setup["ctx"], setup["sol"]
    u, its = ctx.pcg()
    uo, itso, _ = O.pcg(sol.ku, sol.vcycle, m.F[:, 0], m.S.tol, m.S.maxIT)
    f = m.F[:, 0]
    if setup["kind"] == "u_shape":
        # 88 iterations of a tol-1e-3 PCG on the ill-conditioned U: the stopping test may fall one
        # iteration apart, and the solutions then differ by that last step
        assert abs(its - itso) <= 1
        assert abs(f @ u - f @ uo) / abs(f @ uo) < 1e-5
        return
    assert its == itso
    assert _rel(u, uo) < 1e-6
    assert abs(f @ u - f @ uo) / abs(f @ uo) < 1e-8


def test_compliance(setup):
    m, ctx, sol = setup["m"], setup["ctx"], setup["sol"]
    U = np.random.default_rng(4).standard_normal((m.levels[0].numDOFs, 1))
    assert _rel(ctx.unit_compliance(U), O.unit_compliance(m, U)) < 1e-13


@pytest.mark.parametrize("rmin", [np.sqrt(3), 6.0])
def test_filter(setup, rmin):
    m, ctx = setup["m"], setup["ctx"]
    src = np.random.default_rng(6).uniform(0, 1, m.levels[0].numElements)
    out, its = ctx.filter(rmin, src)
    flt = O.PDEFilter(m, rmin, m.S)
    ref = flt(src)
    assert its == flt.last_its
    assert _rel(out, ref) < 1e-10


@pytest.fixture(scope="module")
def mixed_setup():
    from top3d_xl_b200 import Context
    vox = np.ones((12, 24, 12), bool)
    m = O.build_model(vox)
    ctx = Context("mixed")
    ctx.load_voxels(vox)
    x = np.random.default_rng(1).uniform(0.05, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    ctx.set_moduli(E)
    ctx.assemble()
    yield dict(m=m, ctx=ctx, sol=sol)
    ctx.close()


def test_mixed_vcycle_is_fp32_accurate(mixed_setup):
    m, ctx, sol = mixed_setup["m"], mixed_setup["ctx"], mixed_setup["sol"]
    r = np.random.default_rng(3).standard_normal(m.levels[0].numDOFs)
    assert _rel(ctx.vcycle(r), sol.vcycle(r)) < 1e-5


def test_mixed_pcg_keeps_fp64_compliance(mixed_setup):
    # FP32 noise confined to the preconditioner keeps CG's Galerkin property
    m, ctx, sol = mixed_setup["m"], mixed_setup["ctx"], mixed_setup["sol"]
    u, its = ctx.pcg()
    uo, itso, _ = O.pcg(sol.ku, sol.vcycle, m.F[:, 0], m.S.tol, m.S.maxIT)
    f = m.F[:, 0]
    assert abs(its - itso) <= 1
    assert abs(f @ u - f @ uo) / abs(f @ uo) < 1e-6
    assert np.linalg.norm(f - ctx.ku(u)) / np.linalg.norm(f) < m.S.tol


def test_filter_preserves_constants(setup):
    m, ctx = setup["m"], setup["ctx"]
    out, _ = ctx.filter(np.sqrt(3), np.ones(m.levels[0].numElements))
    assert np.max(np.abs(out - 1.0)) < 1e-3


@pytest.mark.parametrize("shape", [(64, 96, 64), (112, 136, 112)])
def test_vcycle_with_large_coarsest_slabs(shape):
    # coarsest grids of 9 x 13 x 9 and 15 x 18 x 15 nodes: elimination trees of several levels,
    # fronts of several 64-wide tiles (Gauss-Jordan steps over many tile tasks)
    from top3d_xl_b200 import Context
    vox = np.ones(shape, bool)
    m = O.build_model(vox)
    x = np.random.default_rng(4).uniform(0.3, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    with Context("fp64") as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        ctx.assemble()
        for seed in (3, 5):  # two solves with the same factors
            r = np.random.default_rng(seed).standard_normal(m.levels[0].numDOFs)
            assert _rel(ctx.vcycle(r), sol.vcycle(r)) < 1e-10
        ctx.assemble()  # a second factorisation through the same scratch and control words
        r = np.random.default_rng(6).standard_normal(m.levels[0].numDOFs)
        assert _rel(ctx.vcycle(r), sol.vcycle(r)) < 1e-10


@pytest.mark.parametrize("kind", ["cuboid", "irregular", "u_shape"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_persistent_coarse_solve_matches_level_launches(kind, precision):
    # the coarsest solve as one dataflow launch (tasks wait for their children's or an ancestor's
    # counters) and as one launch per tree level run the same tasks with the same summation
    # order: the V-cycles agree bit for bit, over repeated solves (the counters are re-armed by
    # each launch) and after a second factorisation.  The U-shaped domain's tree has fronts whose
    # separator holds no present node (nothing eliminated, update DOFs around it): their
    # children's solves up and down must wait past them, for the nearest eliminating ancestor.
    from top3d_xl_b200 import Context
    if kind == "cuboid":
        vox = np.ones((64, 128, 64), bool)
    elif kind == "irregular":
        vox = np.random.default_rng(12).random((64, 128, 64)) < 0.8
        vox[:, 0, :] = True
        vox[:, -1, :] = True
    else:
        vox = np.zeros((64, 160, 64), bool)
        vox[:, :8, :] = True
        vox[:, -8:, :] = True
        vox[:, :, :8] = True
    E = 1.0 + np.random.default_rng(11).uniform(0.0, 1.0, int(vox.sum())) ** 3
    outs = []
    for coop in (1, 0):
        with Context(precision, coarse_coop=coop) as ctx:
            ctx.load_voxels(vox)
            ctx.set_moduli(E)
            ctx.assemble()
            res = []
            for k, seed in enumerate((21, 22, 23)):
                if k == 2:
                    ctx.assemble()
                res.append(ctx.vcycle(np.random.default_rng(seed).standard_normal(ctx.numDOFs)))
            outs.append(res)
    for a, b in zip(*outs):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("kind", ["cuboid", "irregular"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_ku_and_pcg_with_last_row_kernel(kind, precision):
    # y extent a multiple of the K*u tile height (32 nodes): the tile kernel stops one node row
    # short and the grid's last row y = ny runs in its own kernel, in both the plain operator and
    # the PCG step (direction update, stored direction, p'q); fixed DOFs lie on that row too
    from top3d_xl_b200 import Context
    if kind == "cuboid":
        vox = np.ones((32, 20, 12), bool)
    else:
        rng = np.random.default_rng(7)
        vox = rng.random((64, 18, 10)) < 0.8
        vox[:, 0, :] = True
        vox[:, -1, :] = True
    m = O.build_model(vox)
    assert m.levels[0].resY % 32 == 0
    x = np.random.default_rng(8).uniform(0.05, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    with Context(precision) as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        ctx.assemble()
        u = np.random.default_rng(9).standard_normal(m.levels[0].numDOFs)
        assert _rel(ctx.ku(u), sol.ku(u)) < 1e-13
        up, its = ctx.pcg()
    uo, itso, _ = O.pcg(sol.ku, sol.vcycle, m.F[:, 0], m.S.tol, m.S.maxIT)
    f = m.F[:, 0]
    if precision == "fp64":
        assert its == itso
        assert abs(f @ up - f @ uo) / abs(f @ uo) < 1e-8
    else:
        assert abs(its - itso) <= 1
        assert abs(f @ up - f @ uo) / abs(f @ uo) < 1e-6


@pytest.mark.parametrize("kind", ["cuboid", "irregular"])
def test_standard_vcycle(kind):
    # typeVcycle 'Standard' (TX:758-763, 772-777): level-1 and coarse-level K*u inside the
    # V-cycle.  The operator matches at the default omega; PCG runs at omega 0.4, where the cycle
    # is positive definite (at 0.6 it is indefinite and PCG stalls, in the oracle as well)
    from top3d_xl_b200 import Context
    if kind == "cuboid":
        vox = np.ones((12, 24, 12), bool)
    else:
        rng = np.random.default_rng(5)
        vox = rng.random((13, 27, 11)) < 0.75
        vox[:, 0, :] = True
        vox[:, -1, :] = True
    m = O.build_model(vox)
    x = np.random.default_rng(1).uniform(0.05, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    m.S.typeVcycle = "Standard"
    r = np.random.default_rng(3).standard_normal(m.levels[0].numDOFs)
    with Context("fp64", typeVcycle="Standard") as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        ctx.assemble()
        assert _rel(ctx.vcycle(r), sol.vcycle(r)) < 1e-10
    m.S.weightFactorJacobi = 0.4
    with Context("fp64", typeVcycle="Standard", weightFactorJacobi=0.4) as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        ctx.assemble()
        assert _rel(ctx.vcycle(r), sol.vcycle(r)) < 1e-10
        u, its = ctx.pcg()
    uo, itso, _ = O.pcg(sol.ku, sol.vcycle, m.F[:, 0], m.S.tol, m.S.maxIT)
    f = m.F[:, 0]
    assert abs(its - itso) <= 1
    assert abs(f @ u - f @ uo) / abs(f @ uo) < 1e-8


@pytest.mark.parametrize("shape", [(3, 3, 3), (8, 6, 5), (15, 71, 9), (31, 33, 17), (63, 16, 40), (130, 9, 11)])
@pytest.mark.parametrize("holes", [False, True])
def test_ku_tile_edges(shape, holes):
    # K*u tiles: the smallest grid (one tile, one chunk), extents around a tile's height and width,
    # z-chunks with a short last one, several y tiles; with holes the tiles come from the domain's list
    from top3d_xl_b200 import Context
    vox = np.ones(shape, bool)
    if holes:
        vox[:, 1:-1, :] = np.random.default_rng(3).random((shape[0], shape[1] - 2, shape[2])) < 0.7
    m = O.build_model(vox)
    x = np.random.default_rng(1).uniform(0.05, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    u = np.random.default_rng(2).standard_normal(m.levels[0].numDOFs)
    with Context("fp64") as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        assert _rel(ctx.ku(u), sol.ku(u)) < 1e-13


@pytest.mark.parametrize("shape", [(3, 3, 3), (9, 41, 7), (33, 20, 12), (14, 70, 30), (30, 9, 65)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pcg_step_edges(shape, precision):
    # the PCG step's fused passes (the direction formed inside K*u from the residual and the level-2
    # correction, the residual's update with the y pass of its restriction): tiles, chunks and
    # padded rows of odd extents; the bars are test_pcg's, its counts within one (a knife edge of the stop test)
    from top3d_xl_b200 import Context
    vox = np.ones(shape, bool)
    m = O.build_model(vox)
    x = np.random.default_rng(1).uniform(0.3, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    uo, itso, _ = O.pcg(sol.ku, sol.vcycle, m.F[:, 0], m.S.tol, m.S.maxIT)
    f = m.F[:, 0]
    # the oracle against itself with rounding noise in its V-cycle (a 3 x 3 x 3 model amplifies it to 3e-7)
    rng = np.random.default_rng(5)
    un, _, _ = O.pcg(sol.ku, lambda v: sol.vcycle(v) * (1 + 1e-15 * rng.standard_normal(v.shape)), f, m.S.tol, m.S.maxIT)
    env = abs(f @ un - f @ uo) / abs(f @ uo)
    with Context(precision) as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        ctx.assemble()
        r = np.random.default_rng(3).standard_normal(m.levels[0].numDOFs)
        assert _rel(ctx.vcycle(r), sol.vcycle(r)) < (1e-11 if precision == "fp64" else 1e-5)
        u, its = ctx.pcg()
    assert abs(its - itso) <= 1
    if its == itso:
        assert abs(f @ u - f @ uo) / abs(f @ uo) < max(1e-8 if precision == "fp64" else 1e-6, 10 * env)


@pytest.mark.parametrize("shape", [(3, 3, 3), (9, 41, 7), (31, 33, 17), (63, 16, 40), (130, 9, 11)])
@pytest.mark.parametrize("holes", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed32"])
def test_filter_tile_edges(shape, holes, precision):
    # the filter's tiles (odd extents, short chunks, the domain's tile list), in FP64 and with its CG in FP32;
    # FP64: the bar of test_filter.  FP32: the CG stops at 1e-4 of its right-hand side, and its last step may fall
    # one iteration apart
    from top3d_xl_b200 import Context
    vox = np.ones(shape, bool)
    if holes:
        vox[:, 1:-1, :] = np.random.default_rng(3).random((shape[0], shape[1] - 2, shape[2])) < 0.7
    m = O.build_model(vox)
    src = np.random.default_rng(6).uniform(0, 1, m.levels[0].numElements)
    with Context(precision) as ctx:
        ctx.load_voxels(vox)
        for rmin in (np.sqrt(3), 6.0):
            out, its = ctx.filter(rmin, src)
            flt = O.PDEFilter(m, rmin, m.S)
            ref = flt(src)
            if precision == "fp64":
                assert its == flt.last_its
                assert _rel(out, ref) < 1e-10
            else:
                assert abs(its - flt.last_its) <= 1
                assert _rel(out, ref) < 1e-3


@pytest.mark.parametrize("shape", [(32, 64, 40), (40, 64, 40), (8, 8, 200), (31, 40, 17)])
@pytest.mark.parametrize("holes", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_small_coarse_levels(shape, holes, precision):
    # the levels below the first as one cluster launch (one front of at most 320 nodes: 32 x 64 x 40 has 270) and as
    # separate launches (40 x 64 x 40 has 324): both against the oracle's V-cycle, with test_vcycle's bars
    from top3d_xl_b200 import Context
    vox = np.ones(shape, bool)
    if holes:
        vox[:, 1:-1, :] = np.random.default_rng(3).random((shape[0], shape[1] - 2, shape[2])) < 0.7
    m = O.build_model(vox)
    x = np.random.default_rng(1).uniform(0.3, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    with Context(precision) as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        ctx.assemble()
        for seed in (3, 4):
            r = np.random.default_rng(seed).standard_normal(m.levels[0].numDOFs)
            assert _rel(ctx.vcycle(r), sol.vcycle(r)) < (1e-10 if precision == "fp64" else 1e-5)


@pytest.mark.parametrize("shape", [(52, 56, 52), (52, 52, 60)])
@pytest.mark.parametrize("holes", [False, True])
def test_galerkin_group_sizes(shape, holes):
    # 13 x 14 x 13 = 2366 level-2 elements go two to a block, 13 x 13 x 15 = 2535 sixteen (the last block is short);
    # with holes some groups are void, and both have elements with BC-modified templates; test_vcycle's bar
    from top3d_xl_b200 import Context
    vox = np.ones(shape, bool)
    if holes:
        vox[:, 1:-1, :] = np.random.default_rng(5).random((shape[0], shape[1] - 2, shape[2])) < 0.8
        vox[8:40, 8:44, 12:20] = False
    m = O.build_model(vox)
    x = np.random.default_rng(1).uniform(0.3, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    with Context("fp64") as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        ctx.assemble()
        r = np.random.default_rng(3).standard_normal(m.levels[0].numDOFs)
        assert _rel(ctx.vcycle(r), sol.vcycle(r)) < 1e-10


@pytest.mark.parametrize("shape", [(16, 32, 16), (30, 41, 40), (56, 100, 56)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pcg_end_is_one_decision(shape, precision):
    # the kernel that takes the residual pass's sums also ends the solve: all its CTAs and warps have to act alike
    # (one cluster launch, or the restriction of larger grids), with the launches of the chunk that follow
    # doing nothing.  Every sum has a fixed order, so repeated solves are equal bit for bit.
    from top3d_xl_b200 import Context
    vox = np.ones(shape, bool)
    E = np.random.default_rng(1).uniform(0.05, 1.0, vox.size)
    with Context(precision) as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        ctx.assemble()
        u0, its0 = ctx.pcg()
        assert 0 < its0 < 800
        for _ in range(12):
            u, its = ctx.pcg()
            assert its == its0
            assert np.array_equal(u, u0)


@pytest.mark.parametrize("bad", ["start", "moduli"])
@pytest.mark.parametrize("shape,cycle", [((20, 36, 24), "Adapted"), ((50, 100, 50), "Adapted"), ((50, 100, 50), "Standard")])
def test_solve_after_a_nan_solve(shape, cycle, bad):
    # a solve that ends in NaN (a NaN in its start vector or moduli) leaves nothing behind, off the domain either: the next
    # solve on the context is the one that a fresh context computes
    from top3d_xl_b200 import Context
    ny, nx, nz = shape
    vox = np.ones(shape, bool)
    vox[ny // 4:3 * ny // 4, nx // 4:2 * nx // 3, nz // 4:3 * nz // 4] = False
    vox[:, 4 * nx // 5:, nz // 2:] = False
    E = np.random.default_rng(1).uniform(0.05, 1.0, int(vox.sum()))
    with Context("fp64", maxIT=200, typeVcycle=cycle) as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        ctx.assemble()
        u0, its0 = ctx.pcg()
        assert its0 < 200 and np.isfinite(u0).all()
        y0, f0, z0 = ctx.ku(u0), ctx.filter(2.5, E)[0], ctx.vcycle(u0)
        if bad == "start":
            ctx.pcg(np.full(ctx.numDOFs, np.nan))
        else:
            ctx.set_moduli(np.full(E.size, np.nan))
            ctx.assemble()
            ctx.pcg()
            ctx.set_moduli(E)
            ctx.assemble()
        ctx.ku(np.full(ctx.numDOFs, np.nan))
        ctx.filter(2.5, np.full(E.size, np.nan))
        assert np.array_equal(ctx.vcycle(u0), z0)
        u, its = ctx.pcg()
        assert its == its0
        assert np.array_equal(u, u0)
        assert np.array_equal(ctx.ku(u0), y0) and np.array_equal(ctx.filter(2.5, E)[0], f0)


def test_host_copies_before_and_with_the_slots():
    # long copies from and to pageable memory: the first 64 MB go through the runtime, later ones through page-locked
    # slots in chunks of 1 MB (the last one short); both carry every byte, and a new context starts over
    from top3d_xl_b200 import Context
    shape = (64, 96, 72)  # 3.4 MB of densities
    rng = np.random.default_rng(9)
    for _ in range(2):
        with Context("fp64") as ctx:
            ctx.load_voxels(np.ones(shape, bool))
            for k in range(14):  # 6.8 MB each
                x = rng.uniform(0.0, 1.0, ctx.numElements)
                ctx.set_density(x)
                assert np.array_equal(ctx.density(), x), k


@pytest.mark.parametrize("shape", [(56, 48, 56), (52, 56, 52)])
def test_galerkin_blocks_on_both_sides_of_the_line(shape):
    # extents are padded to multiples of 8, level 2 has 14 x 12 x 14 = 2352 elements, just below the line at 2368 (two to a
    # block), or 14 x 14 x 14 = 2744, above it (sixteen to a block, the last one short); groups that are void, and
    # elements with BC-modified templates, in both; test_vcycle's bar
    from top3d_xl_b200 import Context
    vox = np.ones(shape, bool)
    vox[:, 20:40, 12:24] = False  # 14 x 5 level-2 elements in a row of the numbering, three times
    vox[8:30, 4:18, 30:41] = False
    m = O.build_model(vox)
    L2 = m.levels[1]
    n2 = L2.resX * L2.resY * L2.resZ
    assert n2 == {48: 2352, 56: 2744}[shape[1]] and (n2 < 148 * 16) == (shape[1] == 48)
    assert n2 < 148 * 16 or n2 % 16 != 0
    x = np.random.default_rng(1).uniform(0.3, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    with Context("fp64") as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        ctx.assemble()
        for seed in (3, 4):
            r = np.random.default_rng(seed).standard_normal(m.levels[0].numDOFs)
            assert _rel(ctx.vcycle(r), sol.vcycle(r)) < 1e-10


@pytest.mark.parametrize("shape,zlo,zhi", [((31, 48, 63), 10, 49), ((31, 31, 100), 13, 91)])
@pytest.mark.parametrize("precision", ["fp64", "mixed32"])
def test_tile_lists_with_gaps(shape, zlo, zhi, precision):
    # a void larger than a tile along y, x and z, which begins and ends inside z-chunks: the launches of K*u, of the fused
    # PCG step and of the filter take lists with gaps inside the domain, and planes [lo, hi) of a chunk that begin after
    # or end before the chunk's own (for the first shape 48 of 264 K*u tiles are left out, 4 begin late and 16 end early).
    # Bars: test_ku_tile_edges', test_vcycle's and test_filter_tile_edges'; the solve goes to 1e-8, so that its compliance
    # is within 1e-8 of the oracle's (its error is of the order of the residual's square), with counts within a twentieth
    # (a tenth with the preconditioner in FP32)
    from top3d_xl_b200 import Context
    vox = np.ones(shape, bool)
    vox[3:, shape[1] // 5:shape[1] - 5, zlo:zhi] = False
    m = O.build_model(vox)
    x = np.random.default_rng(1).uniform(0.3, 1.0, m.levels[0].numElements)
    S = m.S
    E = S.modulusMin + x ** S.SIMPpenalty * (S.modulus - S.modulusMin)
    sol = O.Solver(m)
    sol.assemble(E)
    f = m.F[:, 0]
    uo, itso, _ = O.pcg(sol.ku, sol.vcycle, f, 1e-8, 800)
    u = np.random.default_rng(2).standard_normal(m.levels[0].numDOFs)
    src = np.random.default_rng(6).uniform(0, 1, m.levels[0].numElements)
    with Context(precision, tol=1e-8) as ctx:
        ctx.load_voxels(vox)
        ctx.set_moduli(E)
        assert _rel(ctx.ku(u), sol.ku(u)) < 1e-13
        ctx.assemble()
        assert _rel(ctx.vcycle(u), sol.vcycle(u)) < (1e-10 if precision == "fp64" else 1e-5)
        ug, its = ctx.pcg()
        assert itso < 800 and abs(its - itso) <= max(1, itso // (20 if precision == "fp64" else 10))
        assert abs(f @ ug - f @ uo) / abs(f @ uo) < 1e-8
    with Context(precision) as ctx:
        ctx.load_voxels(vox)
        for rmin in (np.sqrt(3), 6.0):
            out, its = ctx.filter(rmin, src)
            flt = O.PDEFilter(m, rmin, m.S)
            ref = flt(src)
            if precision == "fp64":
                assert its == flt.last_its
                assert _rel(out, ref) < 1e-10
            else:
                assert abs(its - flt.last_its) <= 1
                assert _rel(out, ref) < 1e-3
