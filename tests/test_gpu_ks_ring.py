"""Staggered rational force with pole counts below, at and above the depth of the
ring that the kernel streams poles and links through, on a checkerboard of 432
sites (13.5 blocks of 32)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DIMS, BC = (6, 4, 6, 6), (1, -1, 1, -1)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 64])
def test_pole_counts(ctx, clg, oracle, n):
    lat = clg.Lattice(ctx, DIMS, BC)
    U, F = clg.CFieldGaugeSU3(lat), clg.CFieldGaugeSU3(lat)
    U.InitialField(clg.GAUGE_HAAR, 91, 1)
    F.InitialField(clg.GAUGE_EXPH, 92, 1, 0.3)
    pi = [clg.CFieldFermionKSSU3(lat, 0.1) for _ in range(n)]
    pd = [clg.CFieldFermionKSSU3(lat, 0.1) for _ in range(n)]
    for k in range(n):
        pi[k].InitialField(clg.SOURCE_GAUSS, 93, 2 + k)
        pd[k].InitialField(clg.SOURCE_GAUSS, 94, 2 + k)
    a = np.linspace(0.2, 1.7, n)
    Uh, F0 = U.CopyDataOut(), F.CopyDataOut()
    clg.CFieldFermionKSSU3.DerivateD0(F, U, pi, pd, a)
    want = oracle.ks_force(DIMS, Uh, [f.to_numpy() for f in pi], [f.to_numpy() for f in pd], a, F=F0, bc=BC)
    # an entry is a sum of 12 n products of magnitude <= max|phi|^2 sum(a), rounded at most
    # 12 n + 8 times: (12 n + 8) 2^-53 of that sum, and once more in the oracle
    top = max(np.abs(f.to_numpy()).max() for f in pi + pd)
    bound = 2 * (12 * n + 8) * 2.0**-53 * 12 * a.sum() * top * top
    assert np.abs(F.CopyDataOut() - want).max() <= bound
