"""Rate smoothing (smooth_photoion_rate.c): the CPU restatement in
oracle/smooth.py against ARGOT's own C built here, bit for bit, with the
reference Makefile's default isolated faces and with periodic faces; and the
CUDA stencil (argot_b200_smooth_rates) against both."""
import numpy as np
import pytest

from conftest import ref_lib
from oracle import smooth as SM


def _rates(edge, seed):
    rng = np.random.default_rng(seed)
    r = (10.0 ** rng.uniform(-16, -9, (6, edge ** 3))).astype(np.float32)
    r[:, rng.random(edge ** 3) < 0.05] = 0.0   # cells that received nothing
    r[3:] *= np.float32(1e-11)                 # heating rates are ~1e-11 of the Gammas
    return r


def _ref(edge, isolated):
    from oracle.oracle import RefLib
    import os
    from oracle import build
    ref_lib(edge)  # skips when no reference build can be had
    path = build.ref_lib_path(edge, isolated=isolated)
    if not os.path.exists(path) and not build.reference_available():
        pytest.skip("reference build unavailable")
    R = RefLib(edge, isolated=isolated)
    R.init(1.0, 1.0, 0.5, 1)
    return R


@pytest.mark.parametrize("isolated", [True, False])
@pytest.mark.parametrize("edge", [16, 32])
def test_restatement_equals_reference(edge, isolated):
    R = _ref(edge, isolated)
    x = _rates(edge, edge + isolated)
    assert np.array_equal(SM.smooth_rates(x, edge, isolated), R.smooth_rates(x))


def test_uniform_field_is_fixed():
    x = np.full((6, 8 ** 3), 3.0e-12, np.float32)
    for iso in (True, False):
        y = SM.smooth_rates(x, 8, iso)
        assert np.allclose(y, x, rtol=1e-6)


def test_entry_point_rejects_bad_arguments():
    import ctypes as C
    from argot_b200 import _lib as L
    from argot_b200.pipeline import unit_box_grid
    lib = L.load()
    g = unit_box_grid(8, 1.0, 1.0)
    assert lib.argot_b200_smooth_rates(C.byref(g), None, None, 1, None) == L.EINVAL
    buf = np.zeros(6 * 8 ** 3, np.float32)
    p = buf.ctypes.data
    assert lib.argot_b200_smooth_rates(C.byref(g), p, p, 1, None) == L.EINVAL   # aliasing
    assert lib.argot_b200_smooth_rates(C.byref(g), p, p + 4, 2, None) == L.EINVAL  # mode


@pytest.mark.gpu
@pytest.mark.parametrize("isolated", [True, False])
@pytest.mark.parametrize("edge", [16, 24, 32])
def test_device_smoothing_bit_identical(cuda_ok, edge, isolated):
    import torch
    from argot_b200 import _lib as L
    from argot_b200.pipeline import unit_box_grid
    import ctypes as C
    lib = L.load()
    g = unit_box_grid(edge, 1.0, 1.0)
    x = _rates(edge, 3 * edge + isolated)
    xin = torch.from_numpy(x.ravel()).cuda()
    out = torch.full_like(xin, -1.0)
    L.check(lib.argot_b200_smooth_rates(C.byref(g), xin.data_ptr(), out.data_ptr(), int(isolated),
                                        torch.cuda.current_stream().cuda_stream), "smooth_rates")
    got = out.view(6, -1).cpu().numpy()
    assert np.array_equal(got, SM.smooth_rates(x, edge, isolated))
    if edge in (16, 32):
        assert np.array_equal(got, _ref(edge, isolated).smooth_rates(x))


def test_dropin_smoothing_rejects_bad_arguments():
    from argot_b200 import _lib as L
    lib = L.load()
    assert lib.argot_b200_set_dropin_smooth_faces(2) == L.EINVAL
    assert lib.argot_b200_set_dropin_smooth_faces(-1) == L.EINVAL
    lib.smooth_photoion_rate(None, None, None, None, None)
    assert lib.argot_b200_last_error() == L.EINVAL
    assert lib.argot_b200_set_dropin_smooth_faces(1) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("isolated", [True, False])
@pytest.mark.parametrize("edge", [16, 24])
def test_dropin_smooth_photoion_rate(cuda_ok, edge, isolated):
    """smooth_photoion_rate with the reference's GPU-build signature: the
    rates of mesh_dev smoothed in place on the device, bit-identical to the
    reference, the same values written to the host mesh, every other field
    left as it was."""
    import ctypes as C
    import torch
    from argot_b200 import _lib as L, abi
    lib = L.load()
    x = _rates(edge, 5 * edge + isolated)
    names = ("GammaHI", "GammaHeI", "GammaHeII", "HeatHI", "HeatHeI", "HeatHeII")
    rng = np.random.default_rng(edge)
    m = np.zeros(edge ** 3, dtype=np.dtype(abi.FluidMesh))
    m["dens"] = rng.uniform(0.5, 2.0, edge ** 3)
    m["chem"]["fHI"] = rng.uniform(0, 1, edge ** 3)
    m["chem"]["GammaHI"] = 7.0
    m["prev_uene"] = 3.0
    for k, n in enumerate(names):
        m["prev_chem"][n] = x[k]
    before = m.copy()
    dev = torch.from_numpy(m.view(np.uint8).copy()).cuda()
    run = abi.RunParam()
    for a in ("x", "y", "z"):
        setattr(run, f"nmesh_{a}_local", edge)
        setattr(run, f"nmesh_{a}_total", edge)
    cp = abi.CudaParam()
    cp.num_cuda_dev = 1
    cp.strm[0] = torch.cuda.current_stream().cuda_stream
    cm = (abi.CudaMemSpace * 1)()
    cm[0].mesh_dev = dev.data_ptr()
    faces = 1 if isolated else 0
    assert lib.argot_b200_set_dropin_smooth_faces(faces) == 0
    try:
        want = SM.smooth_rates(x, edge, isolated)
        host = m.copy()
        lib.smooth_photoion_rate(host.ctypes.data, C.addressof(run), C.addressof(cm), C.addressof(cp), None)
        assert lib.argot_b200_last_error() == 0
        got_dev = dev.cpu().numpy().view(np.dtype(abi.FluidMesh))
        for k, n in enumerate(names):
            assert np.array_equal(got_dev["prev_chem"][n], want[k]), n
            assert np.array_equal(host["prev_chem"][n], want[k]), n
        # nothing else changes, on the device or on the host
        for arr in (got_dev, host):
            for f in ("dens", "chem", "prev_uene"):
                assert np.array_equal(arr[f], before[f])
            for f in ("wmol", "felec", "fHI", "fHII", "fHeI", "fHeII", "fHeIII"):
                assert np.array_equal(arr["prev_chem"][f], before["prev_chem"][f])
        if edge == 16:
            assert np.array_equal(want, _ref(edge, isolated).smooth_rates(x))
        # without a host mesh only the device copy changes (a second pass)
        lib.smooth_photoion_rate(None, C.addressof(run), C.addressof(cm), C.addressof(cp), None)
        assert lib.argot_b200_last_error() == 0
        twice = SM.smooth_rates(want, edge, isolated)
        got2 = dev.cpu().numpy().view(np.dtype(abi.FluidMesh))
        for k, n in enumerate(names):
            assert np.array_equal(got2["prev_chem"][n], twice[k]), n
    finally:
        lib.argot_b200_set_dropin_smooth_faces(1)


def _ragged_planes(n, isolated):
    """Six planes with zeros, subnormals and an infinity, and their smoothing
    in the reference's order of sums."""
    rng = np.random.default_rng(sum(n))
    x = (10.0 ** rng.normal(-12, 3, (6,) + n)).astype(np.float32)
    x[0, rng.random(n) < 0.2] = 0.0
    x[1] *= np.float32(1e-30)
    x[2].flat[n[0] * n[1] * n[2] // 2] = np.inf
    want = np.empty_like(x)
    for s in range(6):
        p = np.pad(x[s], 1, mode="edge" if isolated else "wrap")
        terms = [p[1 + a:1 + a + n[0], 1 + b:1 + b + n[1], 1 + c:1 + c + n[2]]
                 for a in (-1, 0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1)]
        acc = terms[0]
        for t in terms[1:13]:
            acc = acc + t
        d = acc.astype(np.float64) + SM.CENTRAL_WEIGHT * terms[13].astype(np.float64)
        for t in terms[14:]:
            d = d + t.astype(np.float64)
        want[s] = (SM.NORMAL * d).astype(np.float32)
    return x, want


@pytest.mark.gpu
@pytest.mark.parametrize("isolated", [True, False])
@pytest.mark.parametrize("n", [(1, 1, 1), (2, 3, 33), (7, 1, 64), (25, 6, 31), (49, 4, 97), (30, 5, 32), (3, 2, 1)])
def test_device_smoothing_ragged(cuda_ok, n, isolated):
    """Meshes whose axes are no multiple of the kernel's rows, segments and
    32 cells along z, with zeros, subnormals and infinities among the rates:
    the same bits as the restatement."""
    import torch
    from argot_b200 import _lib as L
    import ctypes as C
    x, want = _ragged_planes(n, isolated)
    g = L.Grid(*n, 0, 0, 0, 0.0, 0.0, 0.0, *map(float, n), 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, 1.0, 1.0)
    xin = torch.from_numpy(x.ravel().copy()).cuda()
    out = torch.full_like(xin, -1.0)
    L.check(L.load().argot_b200_smooth_rates(C.byref(g), xin.data_ptr(), out.data_ptr(), int(isolated),
                                             torch.cuda.current_stream().cuda_stream), "smooth_rates")
    assert np.array_equal(out.cpu().numpy().reshape(want.shape), want)


@pytest.mark.gpu
@pytest.mark.parametrize("isolated", [True, False])
@pytest.mark.parametrize("n", [(20000, 1, 1), (1, 9000, 3), (700, 3, 5), (150, 150, 4), (1, 300, 300), (2, 300, 300),
                               (96, 96, 15), (96, 96, 17)])
def test_device_smoothing_thin(cuda_ok, n, isolated):
    """Meshes on both sides of the line between the two kernels: the same
    bits as the restatement."""
    import torch
    from argot_b200 import _lib as L
    import ctypes as C
    x, want = _ragged_planes(n, isolated)
    g = L.Grid(*n, 0, 0, 0, 0.0, 0.0, 0.0, *map(float, n), 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, 1.0, 1.0)
    xin = torch.from_numpy(x.ravel().copy()).cuda()
    out = torch.full_like(xin, -1.0)
    L.check(L.load().argot_b200_smooth_rates(C.byref(g), xin.data_ptr(), out.data_ptr(), int(isolated),
                                             torch.cuda.current_stream().cuda_stream), "smooth_rates")
    assert np.array_equal(out.cpu().numpy().reshape(want.shape), want)


@pytest.mark.gpu
def test_thin_mesh_costs_its_cells(cuda_ok):
    """A mesh of four cells along z takes no longer than one of four times as
    many cells with full rows (measured 58 us and 142 us)."""
    import torch
    from argot_b200 import _lib as L
    import ctypes as C
    lib, st = L.load(), torch.cuda.current_stream().cuda_stream

    def run(n):
        g = L.Grid(*n, 0, 0, 0, 0.0, 0.0, 0.0, *map(float, n), 0.0, 0.0, 0.0, 1.0, 1.0, 1.0, 1.0, 1.0)
        x = torch.rand(6 * n[0] * n[1] * n[2], device="cuda")
        out = torch.empty_like(x)
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(5):
                L.check(lib.argot_b200_smooth_rates(C.byref(g), x.data_ptr(), out.data_ptr(), 1, st), "smooth_rates")
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    assert run((512, 512, 4)) < run((256, 256, 64))
