"""Host- and device-array import / export of links and fields: the tiled reorder
kernels at the edges of their tiles (32 and 64 checkerboard indices), for arrays
aligned to 8 bytes only, against numpy's reordering.  Nothing is computed on the
way, so double-precision data is equal bit for bit."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(2, 2, 2, 2), (2, 4, 2, 4), (4, 6, 2, 10), (4, 4, 4, 8), (6, 2, 14, 4)]


def _device(a, shift):
    """a's bytes on the GPU, `shift` doubles past a 16-byte boundary"""
    import torch

    n = a.size * a.itemsize // 8
    t = torch.zeros(n + 2, dtype=torch.float64, device="cuda")
    t[shift:shift + n] = torch.from_numpy(a.view(np.float64).ravel()).cuda()
    torch.cuda.synchronize()
    return t, C.c_void_p(t.data_ptr() + 8 * shift), n


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("dims", DIMS)
def test_gauge_reorder(ctx, clg, dims, shift):
    rng = np.random.default_rng(5)
    V = int(np.prod(dims))
    a = rng.standard_normal((V, 4, 3, 3)) + 1j * rng.standard_normal((V, 4, 3, 3))
    lat = clg.Lattice(ctx, dims)
    u = clg.CFieldGaugeSU3(lat)
    # Bridge++ order: x fastest
    bridge = np.ascontiguousarray(a.reshape(*dims, 4, 3, 3).transpose(3, 2, 1, 0, 4, 5, 6))
    dev = np.abs(np.einsum("vmik,vmjk->vmij", a, a.conj()) - np.eye(3)).max()
    det = np.abs(np.linalg.det(a) - 1).max()
    for layout, data in ((clg.LAYOUT_CLGBIN, a), (clg.LAYOUT_BRIDGEPP, bridge)):
        u.InitialField(clg.GAUGE_ZERO)
        t, p, n = _device(data, shift)
        assert ctx.lib.clg_gauge_import(u.h, p, layout, 1) == clg.SUCCESS
        np.testing.assert_array_equal(u.CopyDataOut().reshape(a.shape), a)
        np.testing.assert_allclose(u.unitarity(), max(dev, det), rtol=1e-12)
        t.zero_()
        assert ctx.lib.clg_gauge_export(u.h, p, 1) == clg.SUCCESS
        got = t[shift:shift + n].cpu().numpy().view(np.complex128).reshape(a.shape)
        np.testing.assert_array_equal(got, a)
        u.InitialWithByte(data, layout)
        np.testing.assert_array_equal(u.CopyDataOut().reshape(a.shape), a)
    # a NaN anywhere counts as not unitary, and so does an overflow
    for bad in (np.nan, np.inf):
        b = np.broadcast_to(np.eye(3, dtype=np.complex128), a.shape).copy()
        b[V - 1, 3, 2, 1] = bad
        u.InitialWithByte(b)
        assert u.unitarity() >= 1e300
    u.InitialField(clg.GAUGE_IDENTITY)
    assert u.unitarity() == 0.0
    u.InitialField(clg.GAUGE_ZERO)
    assert u.unitarity() == 1.0 and np.abs(u.CopyDataOut()).max() == 0.0


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("subset", ["FULL", "EVEN"])
@pytest.mark.parametrize("kind", ["wilson", "staggered"])
@pytest.mark.parametrize("dims", DIMS)
def test_field_reorder(ctx, clg, dims, kind, subset, shift):
    rng = np.random.default_rng(6)
    V = int(np.prod(dims))
    lat = clg.Lattice(ctx, dims)
    cls, nc = ((clg.CFieldFermionWilsonSquareSU3, (4, 3)) if kind == "wilson" else (clg.CFieldFermionKSSU3, (3,)))
    even = clg.eo_parity(dims) == 0
    # (precision, largest error relative to the site's largest component: half a unit in the last place)
    for prec, tol in ((clg.DOUBLE, 0.0), (clg.SINGLE, 2.0 ** -24), (clg.HALF, 2.0 ** -11 + 2.0 ** -22)):
        f = cls(lat, 0.1, subset=getattr(clg, subset), precision=prec, nrhs=2)
        a = rng.standard_normal((2, V, *nc)) + 1j * rng.standard_normal((2, V, *nc))
        want = a.copy()
        if subset == "EVEN":
            want[:, ~even] = 0
        for r in range(2):
            _, p, n = _device(a[r], shift)
            assert ctx.lib.clg_field_import(f.h, r, p, 1) == clg.SUCCESS
        for r in range(2):
            t, p, n = _device(np.full_like(a[r], 7.0), shift)
            assert ctx.lib.clg_field_export(f.h, r, p, 1) == clg.SUCCESS
            got = t[shift:shift + n].cpu().numpy().view(np.complex128).reshape(want[r].shape)
            np.testing.assert_array_equal(got, f.to_numpy(r))
            d = np.abs((got - want[r]).reshape(V, -1).view(np.float64)).max(1)
            top = np.abs(want[r].reshape(V, -1).view(np.float64)).max(1)
            assert (d <= tol * top).all()


def test_short_device_array_is_refused(ctx, clg):
    """A link array whose allocation ends early is refused on the host (a kernel
    would read or write past it); one that ends with the links is taken."""
    from cuda.bindings import driver, runtime

    lat = clg.Lattice(ctx, (4, 4, 4, 4))
    u = clg.CFieldGaugeSU3(lat)
    u.InitialField(clg.GAUGE_HAAR, 5, 1)
    want, need = u.CopyDataOut(), lat.volume * 4 * 18 * 8
    for size, ok in ((need, True), (need // 2, False)):
        err, p = runtime.cudaMalloc(size)
        assert err == runtime.cudaError_t.cudaSuccess
        attr = driver.CUpointer_attribute.CU_POINTER_ATTRIBUTE_IS_LEGACY_CUDA_IPC_CAPABLE
        err, legacy = driver.cuPointerGetAttribute(attr, p)
        err2, _, held = driver.cuMemGetAddressRange(p)
        known = int(err) == 0 and int(err2) == 0 and legacy and (held < need) != ok
        if known:  # else the host cannot tell that the array is too short
            for call in (lambda: ctx.lib.clg_gauge_export(u.h, C.c_void_p(int(p)), 1),
                         lambda: ctx.lib.clg_gauge_import(u.h, C.c_void_p(int(p)), clg.LAYOUT_CLGBIN, 1)):
                assert (call() == clg.SUCCESS) == ok
            np.testing.assert_array_equal(u.CopyDataOut(), want)
        runtime.cudaFree(p)
        assert known
