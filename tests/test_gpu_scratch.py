"""The context's scratch pool: operators in place and products reuse its blocks,
results do not depend on what a block held before, the pool stays bounded, lets
the longest idle blocks go for new sizes, and gives its memory back when an
allocation fails and when the context ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KAPPA = 0.1355


def test_products_reuse_scratch(clg, oracle):
    import torch

    c = clg.Context(0)
    lat = clg.Lattice(c, (6, 8, 4, 10), (1, 1, 1, -1))
    U = clg.CFieldGaugeSU3(lat)
    U.InitialField(clg.GAUGE_HAAR, 5, 1)
    Uh = U.CopyDataOut()
    for prec, tol in ((clg.DOUBLE, 1e-13), (clg.SINGLE, 2e-6), (clg.HALF, 5e-3)):
        for nrhs in (1, 2):
            a = clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, precision=prec, nrhs=nrhs)
            b = clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, precision=prec, nrhs=nrhs)
            for r in range(nrhs):
                a.InitialField(clg.SOURCE_GAUSS, 9 + r, 2, rhs=r)
            src = [a.to_numpy(r) for r in range(nrhs)]
            a.apply_to(clg.EFO_F_DDdagger, b, U)
            out = [b.to_numpy(r) for r in range(nrhs)]
            a.DDdagger(U)  # in place
            for r in range(nrhs):
                np.testing.assert_array_equal(a.to_numpy(r), out[r])
                want = oracle.wilson_D(lat.dims, Uh, oracle.wilson_D(lat.dims, Uh, src[r], KAPPA, dagger=True), KAPPA)
                assert np.linalg.norm(out[r] - want) <= tol * np.linalg.norm(want)
            a.close()
            b.close()
    # the same calls again allocate nothing
    f = clg.CFieldFermionWilsonSquareSU3(lat, KAPPA)
    f.InitialField(clg.SOURCE_GAUSS, 3, 2)
    f.DDdagger(U)
    f.Dot(f)
    U.plaquette()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info(0)[0]
    for _ in range(3):
        f.DDdagger(U)
        f.D(U)
        f.Dot(f)
        f.norm2()
        U.plaquette()
    assert torch.cuda.mem_get_info(0)[0] == free
    for o in (f, U, lat):
        o.close()
    c.close()


def test_pool_is_bounded_and_given_back(clg):
    import torch

    lib = clg.load_library()
    base = clg.Context(0)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info(0)[0]
    c = clg.Context(0)
    lat = clg.Lattice(c, (32, 32, 32, 16))
    U = clg.CFieldGaugeSU3(lat)
    for nrhs in (1, 2, 4, 8, 14):  # temporaries of 0.1 to 1.4 GB
        f = clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, nrhs=nrhs)
        f.DDdagger(U)
        f.close()
    U.close()
    lat.close()
    c.synchronize()
    held = free0 - torch.cuda.mem_get_info(0)[0]
    assert held <= (1 << 30) + (256 << 20), held  # 1 GB and the context's own scratch
    c.close()
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info(0)[0] <= 64 << 20
    assert lib.clg_context_synchronize(base.h) == clg.SUCCESS
    base.close()


def test_idle_blocks_make_room(clg):
    """Three blocks of 288 MiB fill the pool; a product that then needs 384 MiB
    takes the place of one of them and is kept, so that its next call allocates
    nothing.  An allocation that cannot succeed returns every idle block."""
    import torch

    def held():
        c.synchronize()
        return free0 - torch.cuda.mem_get_info(0)[0]

    c = clg.Context(0)
    lat = clg.Lattice(c, (32, 32, 32, 16))
    U = clg.CFieldGaugeSU3(lat)
    U.InitialField(clg.GAUGE_EXPH, 5, 1, 0.25)
    f = clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, subset=clg.EVEN, nrhs=6)
    g = clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, nrhs=4)
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info(0)[0]
    f.ApplyOperator(clg.OP_MEE_MEEDAG, U)
    three = held()
    assert abs(three - (864 << 20)) <= 16 << 20
    for _ in range(3):
        g.DDdagger(U)
        assert abs(held() - three - (96 << 20)) <= 16 << 20
    with pytest.raises(clg.CLGError):
        clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, nrhs=4000)  # 400 GB
    assert held() <= 16 << 20
    g.DDdagger(U)  # and the context goes on
    for o in (f, g, U, lat):
        o.close()
    c.close()


@pytest.mark.parametrize("init", ["GAUGE_ZERO", "GAUGE_IDENTITY", "GAUGE_HAAR"])
def test_links_are_not_generated_in_a_capture(clg, init):
    """What the links deviate by is noted on the host at once, so a generation that
    a graph would run later is refused and changes nothing."""
    import torch

    s = torch.cuda.Stream()
    c = clg.Context(0, s.cuda_stream)
    lat = clg.Lattice(c, (4, 4, 4, 4))
    U = clg.CFieldGaugeSU3(lat)
    U.InitialField(clg.GAUGE_EXPH, 5, 1, 0.25)
    before, dev = U.CopyDataOut(), U.unitarity()
    t = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="relaxed"):
        t += 1
        status = c.lib.clg_gauge_random(U.h, getattr(clg, init), 1, 1, 0.0)
    assert status != clg.SUCCESS
    graph.replay()
    torch.cuda.synchronize()
    assert U.unitarity() == dev
    np.testing.assert_array_equal(U.CopyDataOut(), before)
    for o in (U, lat):
        o.close()
    c.close()


def test_graphs_outlive_a_larger_reduction(clg, oracle):
    """A solver's captured iterations hold the address of the context's reduction
    buffer: a larger solve on the same context may replace the buffer, and the
    first solver's next call replays on the one it captured."""
    c = clg.Context(0)
    dims = (8, 8, 8, 16)

    def setup(dims, nrhs):
        lat = clg.Lattice(c, dims)
        U = clg.CFieldGaugeSU3(lat)
        U.InitialField(clg.GAUGE_EXPH, 5, 1, 0.25)
        b, x = (clg.CFieldFermionWilsonSquareSU3(lat, KAPPA, nrhs=nrhs) for _ in range(2))
        for r in range(nrhs):
            b.InitialField(clg.SOURCE_GAUSS, 9 + r, 2, rhs=r)
        return lat, U, b, x

    lat, U, b, x = setup(dims, 4)
    for prec in (clg.HALF, clg.DOUBLE):
        S = clg.CSLASolverCG(c, inner_precision=prec, tol_true_rel=1e-10)
        for _ in range(2):
            S.Solve(x, b, U, clg.EFO_F_D)
        first = [x.to_numpy(r) for r in range(4)]
        big = setup((32, 32, 32, 16), 12 if prec == clg.HALF else 24)  # partials for 8192 tiles each
        T = clg.CSLASolverCG(c, inner_precision=clg.HALF, tol_true_rel=1e-10, max_iterations=32)
        T.Solve(big[3], big[2], big[1], clg.EFO_F_D, raise_on_fail=False)
        for o in (T, *reversed(big)):
            o.close()
        x.Zero()
        S.Solve(x, b, U, clg.EFO_F_D)
        for r in range(4):
            np.testing.assert_array_equal(x.to_numpy(r), first[r])
        S.close()
    for o in (x, b, U, lat):
        o.close()
    c.close()
