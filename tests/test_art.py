"""ART diffuse radiation (src/diffuse_photon): the library's angle table and
step-function factors against ARGOT's own setup_diffuse_photon, bit for bit
(CPU); the device kernels and the calc_diffuse_photon_radiation drop-in
against ARGOT's own CPU calc_diffuse_photon_radiation built here (GPU).

The reference adds each ray's I (1 - e^-tau) into its cells in its thread
order; the device does the same sums with float atomics in arbitrary order
and evaluates e^-tau in FP32 where the reference uses double exp/expm1, so
the rates agree to a few float ulps per term, not bit for bit: the tests
hold them to 1e-4 relative (measured: see the assertion messages)."""
import ctypes as C

import numpy as np
import pytest

from conftest import ref_lib

UENETOK = 1.0e4   # uene = 1 <-> T ~ 1e4 K x wmol


def _fields(edge, seed):
    """8 planes: dens, fHI, fHII, fHeI, fHeII, fHeIII, felec, uene (a
    partly ionised lognormal-ish mesh with T in ~[2e3, 5e4] K)"""
    rng = np.random.default_rng(seed)
    n = edge ** 3
    dens = np.exp(rng.normal(0.0, 0.8, n))
    xh = np.clip(rng.beta(0.6, 0.6, n), 1e-4, 1 - 1e-4)
    yhe = rng.dirichlet([1.0, 1.0, 1.0], n)
    felec = xh + 0.0811258278 * (yhe[:, 1] + 2 * yhe[:, 2])
    uene = 10.0 ** rng.uniform(-0.6, 0.8, n)
    return np.stack([dens, 1 - xh, xh, yhe[:, 0], yhe[:, 1], yhe[:, 2], felec, uene]).astype(np.float32)


def _ref(edge):
    R = ref_lib(edge)
    from argot_b200.workload import units
    lunit, denstonh = units()
    R.init(lunit, denstonh, 0.5, 1)
    R.art_init(UENETOK)
    return R, lunit, denstonh


def test_angle_table_and_step_factors_equal_reference():
    from argot_b200 import diffuse as D
    R, _, _ = _ref(16)
    d, bc, c8, st = R.art_table()
    d2, bc2, c82 = D.angle_table(D.NSIDE)
    assert len(d) == 12 * D.NSIDE ** 2
    assert np.array_equal(d, d2) and np.array_equal(bc, bc2) and np.array_equal(c8, c82)
    assert np.array_equal(st, D.step_factors())


def test_angle_table_properties():
    from argot_b200 import diffuse as D
    for nside in (1, 2, 4):
        d, bc, c8 = D.angle_table(nside)
        assert len(d) == 12 * nside ** 2 and c8.sum() == len(d)
        assert np.allclose(np.linalg.norm(d.astype(np.float64), axis=1), 1.0, atol=1e-6)
        # the start face is on the side the dominant component enters from
        face_axis = np.array([2, 2, 0, 0, 1, 1])[bc[:, 0]]
        assert np.all(np.abs(d[np.arange(len(d)), face_axis]) >= np.abs(d).max(axis=1) - 1e-6)
        # processing order: octant, then start face
        key = bc[:, 1] * 8 + bc[:, 0]
        assert np.all(np.diff(key) >= 0)
        # the directions cover the sphere evenly: the mean is ~0
        assert np.abs(d.mean(axis=0)).max() < 1e-6


def test_art_rejects_bad_arguments():
    from argot_b200 import _lib as L
    lib = L.load()
    buf = np.zeros(64, np.float32)
    ibuf = np.zeros(64, np.int32)
    assert lib.argot_b200_art_angle_table(0, buf.ctypes.data, ibuf.ctypes.data, None) == L.EINVAL
    h = C.c_void_p()
    bad = np.array([[0.5, 0.5, 0.7]], np.float32)
    bc = np.array([[6, 0]], np.int32)
    st = np.zeros(6, np.float32)
    assert lib.argot_b200_art_create(bad.ctypes.data, bc.ctypes.data, 1, st.ctypes.data, C.byref(h)) == L.EINVAL
    from argot_b200.pipeline import unit_box_grid
    g = unit_box_grid(8, 1.0, 1.0)
    assert lib.argot_b200_art_rates(None, C.byref(g), 1.0, None, None, None, 1, None, None) == L.EINVAL
    lib.calc_diffuse_photon_radiation(None, None, None, None, None, None, None)
    assert lib.argot_b200_last_error() == L.EINVAL


def _device_rates(edge, planes, lunit, denstonh, apass=None):
    import torch
    from argot_b200 import diffuse as D
    from argot_b200.pipeline import unit_box_grid
    g = unit_box_grid(edge, lunit, denstonh)
    f = torch.from_numpy(planes).cuda()
    r = torch.zeros(6 * edge ** 3, dtype=torch.float32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    art = D.Diffuse()
    art.rates(g, UENETOK, f, r, angles_per_pass=apass, crossings=cnt)
    torch.cuda.synchronize()
    from argot_b200 import _lib as L
    L.check(L.load().argot_b200_check_device_error(torch.cuda.current_stream().cuda_stream), "device error")
    art.close()
    return r.view(6, -1).cpu().numpy(), int(cnt.item())


def _rel(got, want):
    got, want = got.astype(np.float64), want.astype(np.float64)
    scale = np.abs(want).max(axis=1, keepdims=True)
    big = np.abs(want) > 1e-6 * scale
    return (np.abs(got - want)[big] / np.abs(want)[big]).max()


@pytest.mark.gpu
@pytest.mark.parametrize("edge", [16, 24, 32])
def test_art_rates_match_reference(cuda_ok, edge):
    R, lunit, denstonh = _ref(edge)
    planes = _fields(edge, 7 * edge)
    R.art_set_mesh(planes)
    want, _ = R.art_run()
    assert np.isfinite(want).all()
    got, steps = _device_rates(edge, planes, lunit, denstonh)
    assert np.isfinite(got).all()
    err = _rel(got, want)
    assert err < 1e-4, err
    # every direction sends edge^2 rays through the box: at least edge^3
    # ray-cell steps per direction
    assert steps >= 768 * edge ** 3
    # the batch size of angles does not change the result beyond the order
    # of the atomic sums
    got1, steps1 = _device_rates(edge, planes, lunit, denstonh, apass=1)
    assert steps1 == steps
    assert _rel(got1, got) < 1e-5


@pytest.mark.gpu
def test_art_dropin_through_mesh_dev(cuda_ok):
    """calc_diffuse_photon_radiation with the reference's GPU signature: the
    caller's angle table (here the reference's own) and mesh_dev; the
    rates are added to prev_chem, nothing else changes."""
    import torch
    from argot_b200 import _lib as L, abi
    edge = 16
    R, lunit, denstonh = _ref(edge)
    d, bc, c8, st = R.art_table()
    planes = _fields(edge, 99)
    R.art_set_mesh(planes)
    want, _ = R.art_run()
    n = edge ** 3
    m = np.zeros(n, dtype=np.dtype(abi.FluidMesh))
    m["dens"] = planes[0]
    for k, f in enumerate(("fHI", "fHII", "fHeI", "fHeII", "fHeIII", "felec")):
        m["prev_chem"][f] = planes[1 + k]
    m["prev_uene"] = planes[7]
    m["eneg"] = 5.0
    before = m.copy()
    dev = torch.from_numpy(m.view(np.uint8).copy()).cuda()

    class Angle(C.Structure):
        _fields_ = [("xovr", C.c_float), ("yovr", C.c_float), ("zovr", C.c_float),
                    ("base_id", C.c_short), ("corner_id", C.c_short)]

    class Step(C.Structure):
        _fields_ = [("HI", C.c_float * 2), ("HeI", C.c_float * 2), ("HeII", C.c_float * 2)]

    class HostDiffuse(C.Structure):
        _fields_ = [("corner_id_num", C.c_int * 8), ("step_fact", C.POINTER(Step)),
                    ("angle", C.POINTER(Angle))]

    angles = (Angle * len(d))()
    for i in range(len(d)):
        angles[i] = Angle(*d[i].tolist(), int(bc[i, 0]), int(bc[i, 1]))
    step = Step((C.c_float * 2)(*st[0:2]), (C.c_float * 2)(*st[2:4]), (C.c_float * 2)(*st[4:6]))
    hd = HostDiffuse((C.c_int * 8)(*c8.tolist()), C.pointer(step), C.cast(angles, C.POINTER(Angle)))
    run = abi.RunParam()
    for a in ("x", "y", "z"):
        setattr(run, f"nmesh_{a}_local", edge)
        setattr(run, f"nmesh_{a}_total", edge)
        setattr(run, f"delta_{a}", float(np.float32(1.0) / np.float32(edge)))
        setattr(run, f"{a}max", 1.0)
        setattr(run, f"{a}max_local", 1.0)
    run.lunit, run.denstonh, run.uenetok = lunit, denstonh, UENETOK
    cp = abi.CudaParam()
    cp.num_cuda_dev = 1
    cp.strm[0] = torch.cuda.current_stream().cuda_stream
    cm = (abi.CudaMemSpace * 1)()
    cm[0].mesh_dev = dev.data_ptr()
    lib = L.load()
    lib.calc_diffuse_photon_radiation(None, C.addressof(run), C.addressof(cm), C.addressof(cp),
                                      C.addressof(hd), None, None)
    assert lib.argot_b200_last_error() == 0
    got = dev.cpu().numpy().view(np.dtype(abi.FluidMesh))
    names = ("GammaHI", "GammaHeI", "GammaHeII", "HeatHI", "HeatHeI", "HeatHeII")
    rates = np.stack([got["prev_chem"][k] for k in names])
    err = _rel(rates, want)
    assert err < 1e-4, err
    for f in ("dens", "eneg", "chem", "prev_uene"):
        assert np.array_equal(got[f], before[f])
    for f in ("fHI", "fHII", "fHeI", "fHeII", "fHeIII", "felec"):
        assert np.array_equal(got["prev_chem"][f], before["prev_chem"][f])


# ------------------------------------------------ the march in 64 bits
def _march_f64(n, d, lunit, ab, S, dirs, faces):
    """J_s = sum over directions of (sum over rays of I (1 - e^-tau)) /
    (a_s sum of chords) + S_s per cell, float64: parallel rays from the cells
    of each direction's start face, wrapped through the side faces with I
    reset (ray_tracing.c, one isolated rank)."""
    off = (0.521212345, 0.508512345, 0.468287655)
    J = np.zeros(tuple(n) + (3,))
    for o, base in zip(dirs.astype(np.float64), faces):
        ax = (2, 2, 0, 0, 1, 1)[base]
        p, q = [k for k in range(3) if k != ax]
        num, chord = np.zeros(tuple(n) + (3,)), np.zeros(tuple(n))
        for a in range(n[p]):
            for b in range(n[q]):
                i = [0, 0, 0]
                i[p], i[q], i[ax] = a, b, (0 if base % 2 == 0 else n[ax] - 1)
                x = [(i[k] + off[k]) * d[k] for k in range(3)]
                x[ax] = 0.0 if base % 2 == 0 else n[ax] * d[ax]
                nxt = [((i[k] + (o[k] > 0)) * d[k] - x[k]) / o[k] for k in range(3)]
                I, s = np.zeros(3), 0.0
                while True:
                    m = min(nxt)
                    c, idx = (m - s) * lunit, tuple(i)
                    e = -np.expm1(-ab[idx] * c)
                    num[idx] += I * e
                    chord[idx] += c
                    I = I * (1 - e) + S[idx] * e
                    s = m
                    for k in range(3):
                        if nxt[k] == m:
                            nxt[k] += d[k] / abs(o[k])
                            i[k] += 1 if o[k] > 0 else -1
                    if not 0 <= i[ax] < n[ax]:
                        break
                    for k in (p, q):
                        if not 0 <= i[k] < n[k]:
                            i[k] %= n[k]
                            I = np.zeros(3)
        J += num / (ab * np.where(chord > 0, chord, np.inf)[..., None]) + S
    return J


def _unit(v):
    v = np.asarray(v, np.float64)
    return (v / np.linalg.norm(v, axis=-1, keepdims=True)).astype(np.float32)


_SWEPT = ([[1, 1.7, 3], [-0.4, 0.2, -2], [2, 1, 0.9], [-3, 0.3, 2.9], [0.2, 3, -1.1], [0.1, -3, 2], [1e-20, 1e-9, 1],
           [1, 1, 1]], [0, 1, 2, 3, 4, 5, 0, 2])


@pytest.mark.gpu
@pytest.mark.parametrize("n,cell,tol", [((5, 7, 9), (1.0, 1.0, 1.0), 5e-6), ((8, 6, 4), (1.0, 0.7, 1.4), 5e-6),
                                        ((1, 3, 33), (1.0, 1.0, 1.0), 5e-6), ((17, 40, 2), (0.5, 1.0, 1.3), 5e-6),
                                        ((1, 1, 600), (1.0, 1.0, 1.0), 2e-3)])
def test_art_rates_against_f64_march(cuda_ok, n, cell, tol):
    """Swept directions (every start face, a tie, directions along an axis)
    on ragged meshes with uneven cells against the float64 march.  The paths
    are formed in double; what is left is FP32 arithmetic along up to 70
    cells: 5e-6.  On the mesh of 600 cells one direction has a path longer
    than a CTA holds and takes the general march beside the swept ones; its
    float positions are good to 2^-15 of a cell there, a chord is a fraction
    of one, and they add up along the path: 2e-3."""
    import torch
    from argot_b200 import _lib as L, diffuse as D
    vec, faces = _SWEPT
    if n[2] == 600:
        vec, faces = vec + [[3, 2.9, 1]], faces + [0]
    dirs = _unit(vec)
    box = [float(np.float32(a * b)) for a, b in zip(n, cell)]
    from argot_b200.workload import units
    lunit, denstonh = units()
    lunit /= max(box)
    g = L.Grid(*n, 0, 0, 0, 0.0, 0.0, 0.0, *box, 0.0, 0.0, 0.0, *cell, lunit, denstonh)
    nc = int(np.prod(n))
    rng = np.random.default_rng(nc)
    planes = np.stack([_fields(1, int(rng.integers(1 << 30)))[:, 0] for _ in range(nc)], 1)
    bc = np.zeros((len(faces), 2), np.int32)
    bc[:, 0] = faces
    art = D.Diffuse(table=(dirs, bc, None))
    got = torch.zeros(6 * nc, dtype=torch.float32, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    f = torch.from_numpy(planes).cuda()
    for crossings in (None, cnt):
        got.zero_()
        art.rates(g, UENETOK, f, got, crossings=crossings)
    L.check(L.load().argot_b200_check_device_error(torch.cuda.current_stream().cuda_stream), "device error")
    ab, S = _coefficients(planes.astype(np.float64), denstonh)
    J = _march_f64(n, [float(np.float32(c)) for c in cell], lunit, ab.reshape(tuple(n) + (3,)),
                   S.reshape(tuple(n) + (3,)), dirs, faces).reshape(nc, 3) / len(faces)
    st = D.step_factors().astype(np.float64)
    want = np.stack([(J @ [1, 1.128855608262e-01, 5.288790581895e-03]) * st[0], (J @ [0, 1, 1.2404369898e-01]) * st[2],
                     J[:, 2] * st[4], (J @ [1, 3.1154224364e+00, 5.2452188546e-01]) * st[1],
                     (J @ [0, 1, 8.7872474963e+00]) * st[3], J[:, 2] * st[5]])
    err = np.abs(got.view(6, -1).double().cpu().numpy() - want) / np.abs(want)
    assert err.max() < tol, err.max(axis=1)
    # every ray of a swept direction crosses at least one cell per layer
    assert int(cnt.item()) >= sum(nc for _ in _SWEPT[1])
    art.close()


@pytest.mark.gpu
def test_art_many_swept_directions_beside_general_ones(cuda_ok):
    """12288 swept directions and one that takes the general march (its path
    is longer than a CTA holds): the mean of the two passes by themselves.
    The sums of 128 directions are closed one after another, so that what
    rounds is some 100 FP32 additions and as many groups, 6e-8 sqrt(100) at
    most; all 12288 in one FP32 sum would be off by 6e-8 sqrt(2 12288 / 3),
    5e-6."""
    import torch
    from argot_b200 import _lib as L, diffuse as D
    from argot_b200.workload import units
    n = (2, 2, 700)
    lunit, denstonh = units()
    cell = float(np.float32(1.0 / 700))
    box = [float(np.float32(k) * np.float32(cell)) for k in n]
    g = L.Grid(*n, 0, 0, 0, 0.0, 0.0, 0.0, *box, 0.0, 0.0, 0.0, cell, cell, cell, lunit, denstonh)
    nc = int(np.prod(n))
    rng = np.random.default_rng(5)
    f = torch.from_numpy(np.stack([_fields(1, int(rng.integers(1 << 30)))[:, 0] for _ in range(nc)], 1)).cuda()
    dirs, bc, _ = D.angle_table(32)
    long_dir, long_bc = _unit([[3, 2.9, 1]]), np.zeros((1, 2), np.int32)

    def run(d, b):
        art = D.Diffuse(table=(d, b, None))
        r = torch.zeros(6 * nc, dtype=torch.float32, device="cuda")
        art.rates(g, UENETOK, f, r)
        L.check(L.load().argot_b200_check_device_error(torch.cuda.current_stream().cuda_stream), "device error")
        art.close()
        return r.double()

    swept, general = run(dirs, bc), run(long_dir, long_bc)
    both = run(np.concatenate([dirs, long_dir]), np.concatenate([bc, long_bc]))
    want = (len(dirs) * swept + general) / (len(dirs) + 1)
    assert torch.isfinite(want).all() and (want > 0).all()
    err = (both - want) / want
    assert err.square().mean().sqrt() < 6e-7


def _coefficients(f, denstonh):
    """Absorption [cm^-1] and source functions of the three frequencies
    (calc_rmesh_data.c:33-111, diffuse_chemistry.c:13-103) in float64."""
    dens, hi, hii, hei, heii, heiii, fe, u = f
    he = 0.0811258278
    t = np.maximum(u * UENETOK / ((1 + fe) * 0.755 + 0.25 * 0.245), 1.0)
    nh = dens * denstonh
    ne = nh * (hii + he * (heii + 2 * heiii))

    def sig(s, v):
        thr = (1.0, 1.8125, 4.0)[s]
        if s == 1:
            return 7.83e-18 * (1.66 * (v / thr) ** -2.05 - 0.66 * (v / thr) ** -3.05)
        e = np.sqrt(v / thr - 1.0)
        return 6.3e-18 * (1.0, 0, 64.0)[s] / v ** 4 * np.exp(4 - 4 * np.arctan(e) / e) / (1 - np.exp(-2 * np.pi / e))

    cs = [float(np.float32(sig(s, (1.0, 1.8125, 4.0)[s] + 1e-7))) for s in range(3)]
    k = [cs[0] * hi * nh, cs[1] * he * hei * nh, cs[2] * he * heii * nh]
    ab = np.stack([k[0], k[0] * 1.9529766579e-01 + k[1], k[0] * 1.9513732355e-02 + k[1] * 2.6858709594e-01 + k[2]], -1)
    ab = ab + 1e-31
    l, tev = np.log(t * 8.61623e-5), t * 8.61623e-5
    p = np.polyval([-3.071135243196595e-9, -1.856767039775261e-8, 5.755614137575758e-7, 4.989108920299513e-6,
                    -0.00001421502914054107, -0.0003212605213188796, -0.002380861877349834, -0.02026044731984691,
                    -0.7241125657826851, -28.61303380689232], l)

    def b(lam, a):
        return a * lam ** 1.5 / (1 + (lam / 2.740) ** 0.407) ** 2.242

    low = 3.92e-13 / tev ** 0.6353
    hot = 1.54e-9 * (1 + 0.3 / np.exp(8.099328789667 / tev)) / (np.exp(40.49664394833662 / tev) * tev ** 1.5)
    he2a = np.where(tev > 0.8, hot + low, low)
    he2b = np.where(t > 500.3, 1.26e-14 * (2 * 285335.0 / t) ** 0.75, (1.12e-10 - 2.1e-11 * np.log10(t)) / np.sqrt(t))
    he3a = 3.36e-10 / np.sqrt(t) / (t / 1e3) ** 0.2 / (1 + (t / 1e6) ** 0.7)
    rec = (np.exp(p) - b(2 * 157807.0 / t, 2.753e-14), he2a - he2b, he3a - b(2 * 631515.0 / t, 1.3765e-14))
    ion = (hii * nh, he * heii * nh, he * heiii * nh)
    e = np.stack([r * ne * x * 13.6 * w * 1.6022e-12 / (4 * np.pi) for r, x, w in zip(rec, ion, (1.0, 1.8125, 4.0))], -1)
    return ab, e / ab
