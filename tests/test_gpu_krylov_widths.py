"""GMRES and multi-shift FOM / GMRES at Krylov dimensions around the group size
of the multi-dot launches (4 inner products per block) and at the limits, on a
lattice whose checkerboard is no multiple of a block, GMRES on both sides of the
size from which one block takes all columns, and in a batch of uneven lattices:
solutions to the oracle's true residual 1e-10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KAPPA, DIMS, TOL = 0.1355, (4, 6, 4, 10), 1e-10


def _setup(clg, ctx, nrhs=1):
    lat = clg.Lattice(ctx, DIMS)
    U = clg.CFieldGaugeSU3(lat)
    U.InitialField(clg.GAUGE_HAAR, 0xC1A60001, 1)
    b = clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, nrhs=nrhs)
    for r in range(nrhs):
        b.InitialField(clg.SOURCE_GAUSS, 50 + r, 2, rhs=r)
    return lat, U, b


@pytest.mark.parametrize("max_dim", [1, 3, 4, 5, 8, 16])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_gmres_widths(ctx, clg, oracle, max_dim, prec):
    lat, U, b = _setup(clg, ctx, 3)
    x = clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, nrhs=3)
    infos = clg.CSLASolverGMRES(ctx, inner_precision=prec, MaxDim=max_dim).Solve(x, b, U, clg.EFO_F_D)
    op = oracle.Operator("WILSON_D", DIMS, U.CopyDataOut(), KAPPA)
    for r in range(3):
        assert infos[r]["status"] == 0
        assert op.true_residual(b.to_numpy(r), x.to_numpy(r)) <= TOL


# 16384 sites over all right-hand sides is the last size of the grouped form:
# 8^4 with 8 and 9 of them, and 20160 on a checkerboard of 5040 sites (19.7 blocks)
@pytest.mark.parametrize("dims,nrhs", [((8, 8, 8, 8), 8), ((8, 8, 8, 8), 9), ((6, 10, 14, 12), 4)])
@pytest.mark.parametrize("max_dim", [1, 4, 5, 16])
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_gmres_forms(ctx, clg, oracle, dims, nrhs, max_dim, prec):
    lat = clg.Lattice(ctx, dims)
    U = clg.CFieldGaugeSU3(lat)
    U.InitialField(clg.GAUGE_HAAR, 0xC1A60001, 1)
    b, x = (clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, nrhs=nrhs) for _ in range(2))
    for r in range(nrhs):
        b.InitialField(clg.SOURCE_GAUSS, 50 + r, 2, rhs=r)
    S = clg.CSLASolverGMRES(ctx, inner_precision=prec, MaxDim=max_dim)
    infos = S.Solve(x, b, U, clg.EFO_F_D)
    op = oracle.Operator("WILSON_D", dims, U.CopyDataOut(), KAPPA)
    for r in range(nrhs):
        assert infos[r]["status"] == 0
        assert op.true_residual(b.to_numpy(r), x.to_numpy(r)) <= TOL
    for o in (S, b, x, U, lat):
        o.close()


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_gmres_batch_skips_padding(ctx, clg, oracle, prec):
    """Eight 4^4 lattices beside one of 24^3x16 hold 1 % of its sites: solved in
    one call they may not cost as if each were padded to it (3 to 4 times the
    large one alone; 1.3 times where the padding is skipped)."""
    import time

    def batch(dims_list):
        lats = [clg.Lattice(ctx, d) for d in dims_list]
        us = [clg.CFieldGaugeSU3(lat) for lat in lats]
        bs, xs = ([clg.CFieldFermionWilsonSquareSU3(lat, KAPPA) for lat in lats] for _ in range(2))
        for i, (u, b) in enumerate(zip(us, bs)):
            u.InitialField(clg.GAUGE_HAAR, 0xC1A60001 + i, 1)
            b.InitialField(clg.SOURCE_GAUSS, 50 + i, 2)
        S = clg.CSLASolverGMRES(ctx, inner_precision=prec, MaxDim=12)
        best = 1e9
        for _ in range(5):
            ctx.synchronize()
            t = time.perf_counter()
            infos = S.SolveLattices(xs, bs, us, clg.EFO_F_D)
            best = min(best, time.perf_counter() - t)
        for lat, u, b, x, i in zip(lats, us, bs, xs, infos):
            op = oracle.Operator("WILSON_D", lat.dims, u.CopyDataOut(), KAPPA)
            assert i["status"] == 0 and op.true_residual(b.to_numpy(), x.to_numpy()) <= TOL
        for o in (S, *bs, *xs, *us, *lats):
            o.close()
        return best

    alone = batch([(24, 24, 24, 16)])
    assert batch([(24, 24, 24, 16)] + 8 * [(4, 4, 4, 4)]) <= 2 * alone


@pytest.mark.parametrize("solver,max_dim", [("FOM", 2), ("FOM", 4), ("FOM", 5), ("FOM", 32), ("GMRES", 3),
                                            ("GMRES", 5), ("GMRES", 32)])
def test_multishift_widths(ctx, clg, oracle, solver, max_dim):
    lat, U, b = _setup(clg, ctx)
    shifts = [2.0, 0.5, 1j, 0.5 + 0.5j, 1 - 1j]
    xs = [clg.CFieldFermionWilsonSquareSU3(lat, KAPPA) for _ in shifts]
    S = getattr(clg, "CMultiShift" + solver)(ctx, MaxDim=max_dim)
    op = oracle.Operator("WILSON_D", DIMS, U.CopyDataOut(), KAPPA)
    for _ in range(2):  # the second call reuses the basis and its device state
        infos = S.Solve(xs, shifts, b, U, clg.EFO_F_D)
        for k, s in enumerate(shifts):
            assert infos[k]["status"] == 0
            assert op.true_residual(b.to_numpy(), xs[k].to_numpy(), complex(s)) <= TOL
    # a zero right-hand side has the zero solution
    b.Zero()
    S.Solve(xs, shifts, b, U, clg.EFO_F_D)
    assert max(np.abs(x.to_numpy()).max() for x in xs) == 0.0
