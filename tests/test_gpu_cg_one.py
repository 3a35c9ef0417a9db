"""CG on one Wilson source: the sums that the next kernel adds up itself, on both
sides of the partial count from which they are folded first, and a breakdown in
(p, A p)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KAPPA = 0.1355


def _context(clg, cfg=None, **env):
    old = {k: os.environ.get(k) for k in ("CLG_HOP_CONFIG", *env)}
    os.environ.update({k: v for k, v in {"CLG_HOP_CONFIG": cfg, **env}.items() if v})
    try:
        return clg.Context(0)
    finally:
        for k, v in old.items():
            os.environ.pop(k, None)
            if v is not None:
                os.environ[k] = v


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_partials_are_folded(clg, oracle, prec):
    """This lattice leaves 576 partials from blocks of 256 threads and 2304 from
    blocks of 64: above 2048 every iteration has one launch more, which folds them."""
    dims, count = (16, 16, 32, 36), []
    for cfg in ("0:256", "0:64"):
        c = _context(clg, cfg)
        lat = clg.Lattice(c, dims)
        U = clg.CFieldGaugeSU3(lat)
        U.InitialField(clg.GAUGE_EXPH, 0xC1A60001, 1, 0.25)
        b, x = (clg.CFieldFermionWilsonSquareSU3(lat, KAPPA) for _ in range(2))
        b.InitialField(clg.SOURCE_GAUSS, 400, 2)
        S = clg.CSLASolverCG(c, inner_precision=prec, tol_true_rel=1e-10)
        k0 = c.kernel_count()
        info = S.Solve(x, b, U, clg.EFO_F_D)[0]
        count.append((c.kernel_count() - k0, info["iterations"] // 2))
        assert info["status"] == 0
        ref = oracle.Operator("WILSON_D", dims, U.CopyDataOut(), KAPPA)
        assert ref.true_residual(b.to_numpy(), x.to_numpy()) <= 1e-10
        for o in (S, b, x, U, lat):
            o.close()
        c.close()
    (few, n0), (many, n1) = count
    assert abs(n0 - n1) <= 8 and many - few >= n1 // 2


@pytest.mark.parametrize("cfg", [None, "0:128"])
def test_breakdown_counts_its_iteration(clg, cfg):
    """Links of 1e13 are finite in single precision and (p, A p) is not: the solve
    ends with a breakdown, at the same count of applications as the iteration with
    separate sums, and leaves a finite solution."""
    dims, got = (8, 8, 8, 8), []
    for fused in ("1", "0"):
        c = _context(clg, cfg, CLG_FUSED_CG=fused)
        lat = clg.Lattice(c, dims)
        U = clg.CFieldGaugeSU3(lat)
        U.InitialField(clg.GAUGE_HAAR, 0xC1A60001, 1)
        U.InitialWithByte(1e13 * U.CopyDataOut())
        b, x = (clg.CFieldFermionWilsonSquareSU3(lat, KAPPA) for _ in range(2))
        b.InitialField(clg.SOURCE_GAUSS, 400, 2)
        S = clg.CSLASolverCG(c, inner_precision=clg.SINGLE, tol_true_rel=1e-10)
        info = S.Solve(x, b, U, clg.EFO_F_D, raise_on_fail=False)[0]
        got.append((info["status"], info["iterations"], info["outer"], bool(np.isfinite(x.to_numpy()).all())))
        for o in (S, b, x, U, lat):
            o.close()
        c.close()
    assert got[0] == got[1]
    assert got[0][0] != 0 and got[0][1] > 0 and got[0][3]
