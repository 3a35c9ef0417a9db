"""Full-lattice forms of D (both checkerboards in one launch, with and without
chunks of y-rows) and the four-threads-per-site form, pinned through the tune
file, against two one-thread-per-site checkerboard hops of the same operator.
The arithmetic per site is the same in the same order, so FP64 and FP16 results
are equal bit for bit; FP32 to 2e-6 (the compiler may contract the rebuilt link
row's products differently per kernel, a few units of 2^-24 on sums of 24)."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KAPPA = 0.1355


def _context(clg, tmp_path, lines):
    path = str(tmp_path / "tune.txt")
    with open(path, "w") as f:
        f.write("".join(f"{k}={v}\n" for k, v in lines.items()))
    old = os.environ.get("CLG_TUNE_FILE")
    os.environ["CLG_TUNE_FILE"] = path
    try:
        return clg.Context(0)
    finally:
        if old is None:
            del os.environ["CLG_TUNE_FILE"]
        else:
            os.environ["CLG_TUNE_FILE"] = old


def _key(kind, prec, dagger, dims, nrhs):
    name = "wilson" if kind == "wilson" else "ks"
    return f"{name}_p{prec}_d{dagger}_V{int(np.prod(dims)) // 2}_n{nrhs}_r{12 if prec == 1 else 0}"


def _cfg(block, variant):
    return block | (variant << 16)


FULL = [_cfg(64, 32), _cfg(256, 33), _cfg(128, 34), _cfg(64, 35), _cfg(128, 36)]
MID = [_cfg(64, 40), _cfg(64, 42)]  # FP64 Wilson


# the last one is cut into chunks of 16 y-rows in double precision
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (6, 10, 14, 12), (4, 64, 32, 32)])
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("kind", ["wilson", "staggered"])
def test_full_forms(clg, tmp_path, kind, prec, dims):
    big = np.prod(dims) > 1 << 16
    for nrhs in (1,) if big else (1, 3):
        outs = []
        for cfg in [0] + FULL + (MID if kind == "wilson" and prec == 0 else []):
            if kind == "staggered" and cfg == FULL[-1]:
                continue
            dags = (0, 1) if kind == "wilson" else (0,)
            keys = [_key(kind, prec, d, dims, nrhs) for d in dags]
            # the checkerboard hops that form 0 launches: one thread per site
            plain = {k + auto: _cfg(128, 0) for k in keys for auto in ("", "_auto")}
            c = _context(clg, tmp_path, {**plain, **{k + "_full": cfg for k in keys}})
            lat = clg.Lattice(c, dims, (1, -1, 1, -1))
            U = clg.CFieldGaugeSU3(lat)
            U.InitialField(clg.GAUGE_EXPH, 0xC1A60001, 1, 0.25)
            cls = clg.CFieldFermionWilsonSquareSU3 if kind == "wilson" else clg.CFieldFermionKSSU3
            f, g = (cls(lat, KAPPA, precision=prec, nrhs=nrhs) for _ in range(2))
            for r in range(nrhs):
                f.InitialField(clg.SOURCE_GAUSS, 300 + r, 2, rhs=r)
            res = []
            for op in (clg.EFO_F_D, clg.EFO_F_Ddagger):
                f.apply_to(op, g, U, clg.EOCT_Real, 0.5)
                res += [g.to_numpy(r) for r in range(nrhs)]
            outs.append(res)
            for o in (f, g, U, lat):
                o.close()
            c.close()
        for res in outs[1:]:
            for got, want in zip(res, outs[0]):
                if prec == 1:
                    assert np.linalg.norm(got - want) <= 2e-6 * np.linalg.norm(want)
                else:
                    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("dims", [(2, 4, 2, 2), (6, 10, 14, 12)])
def test_split_hop(clg, tmp_path, dims, prec):
    outs = []
    for cfg in (_cfg(128, 0), _cfg(128, 4)):
        c = _context(clg, tmp_path, {_key("wilson", prec, d, dims, 1): cfg for d in (0, 1)})
        lat = clg.Lattice(c, dims)
        U = clg.CFieldGaugeSU3(lat)
        U.InitialField(clg.GAUGE_EXPH, 0xC1A60001, 1, 0.25)
        f = clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, subset=clg.EVEN, precision=prec)
        f.InitialField(clg.SOURCE_GAUSS, 300, 2)
        f.ApplyOperator(clg.OP_MEE, U)
        f.ApplyOperator(clg.OP_MEE_DAG, U)
        outs.append(f.to_numpy())
        for o in (f, U, lat):
            o.close()
        c.close()
    if prec == 1:
        assert np.linalg.norm(outs[1] - outs[0]) <= 2e-6 * np.linalg.norm(outs[0])
    else:
        np.testing.assert_array_equal(outs[1], outs[0])


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_split_cg_epilogues(clg, oracle, tmp_path, prec):
    """the fused CG iteration on the four-threads-per-site epilogues, with a
    partial last block (5040 sites per checkerboard), to the oracle's residual"""
    dims, n = (6, 10, 14, 12), 1 if prec == 2 else 2
    c = _context(clg, tmp_path, {_key("wilson", prec, d, dims, n): _cfg(128, 4) for d in (0, 1)})
    lat = clg.Lattice(c, dims)
    U = clg.CFieldGaugeSU3(lat)
    U.InitialField(clg.GAUGE_EXPH, 0xC1A60001, 1, 0.25)
    b, x = (clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, nrhs=n) for _ in range(2))
    for r in range(n):
        b.InitialField(clg.SOURCE_GAUSS, 400 + r, 2, rhs=r)
    for op, name in ((clg.EFO_F_D, "WILSON_D"), (clg.EFO_F_Ddagger, "WILSON_DDAG")):
        infos = clg.CSLASolverCG(c, inner_precision=prec, tol_true_rel=1e-10).Solve(x, b, U, op)
        ref = oracle.Operator(name, dims, U.CopyDataOut(), KAPPA)
        for r in range(n):
            assert infos[r]["status"] == 0
            assert ref.true_residual(b.to_numpy(r), x.to_numpy(r)) <= 1e-10
