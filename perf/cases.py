"""The work this framework does for its users, as cases to be timed and compared.

Kinds of case, each through public entry points:

* ``step``: one radiation iteration of the point-source path on one mesh: the
  fields packed again (the chemistry between iterations changes the ionised
  fractions), rays generated, columns marched, rates integrated.  Small and
  ordinary meshes run the calls in sequence, large ones in parts on two
  streams, as the benchmark does.  ``f32`` rates on compensated columns, or
  ``f64`` rates on reference-order columns (the reference's own algorithm).
* ``surrogate``: the same iteration with the learned frequency integral.
* ``batch``: many problems of uneven size in one captured graph.
* ``segments``: explicit ray segments marched and stitched into light rays.
* ``smooth``: the 27-point smoothing of the six rate fields.
* ``diffuse``: the diffuse-radiation pass over 768 directions.

Inputs are synthetic, drawn from the seed: lognormal meshes with ionised
regions around the sources, neutral meshes, and fully ionised ones.
``exact`` restates every path but the largest in float64 torch.
"""
import ctypes as C
import math

import numpy as np
import torch

from argot_b200 import _lib as L
from argot_b200.batch import Batch
from argot_b200.diffuse import Diffuse
from argot_b200.pipeline import Problem, unit_box_grid
from argot_b200.surrogate import Surrogate
from argot_b200.workload import Workload

LUNIT = 6.6e-3 * 3.086e24   # 6.6 kpc box [cm]
DENSTONH = 1.0e-3           # code density 1 = 1e-3 hydrogen atoms per cm^3
HE = 0.0811258278           # helium atoms per hydrogen atom
THETA = 0.5                 # oct-tree opening angle
UENETOK = 1.0e4             # internal energy -> temperature
THR = (1.0, 1.8125, 4.0)    # ionisation thresholds [HI Lyman limits]
H_NUL = 6.626e-27 * 3.28e15
TEMP = 1.0e5                # blackbody sources


def listed():
    return [
        # a unit-test sized problem: launches and latency count
        dict(name="step_32", kind="step", edge=32, nsrc=8, mesh="tanh", sigma=1.0, clustered=False, mode="f32",
             overlap=0),
        # the plain benchmark problem: uniform neutral mesh, 16 sources
        dict(name="step_64_neutral", kind="step", edge=64, nsrc=16, mesh="neutral", sigma=0.0, clustered=False,
             mode="f32", overlap=0),
        # a ragged mesh through the reference's own algorithm (reference-order columns, FP64 rates)
        dict(name="step_75_f64", kind="step", edge=75, nsrc=24, mesh="tanh", sigma=1.0, clustered=False,
             mode="f64", overlap=0),
        # the precision benchmark problem, in overlapped parts
        dict(name="step_128", kind="step", edge=128, nsrc=256, mesh="tanh", sigma=1.0, clustered=False, mode="f32",
             overlap=8),
        # a production-sized mesh with clustered sources, in overlapped parts
        dict(name="step_256", kind="step", edge=256, nsrc=1024, mesh="tanh", sigma=1.2, clustered=True, mode="f32",
             overlap=32),
        # late reionisation: everything ionised, most rays served by the network
        dict(name="surrogate_96", kind="surrogate", edge=96, nsrc=128, mesh="ionized", sigma=1.0, clustered=False),
        # an ensemble of uneven problems in one graph
        dict(name="batch_8", kind="batch", nprob=8, emin=32, emax=96, smax=256, sigma=1.0),
        # a large list of explicit segments, up to three per light ray
        dict(name="segments_128", kind="segments", edge=128, nray=500_000, precision="kahan", sigma=1.0),
        # smoothing between iterations: a small periodic mesh, a large isolated one
        dict(name="smooth_50", kind="smooth", edge=50, isolated=False),
        dict(name="smooth_256", kind="smooth", edge=256, isolated=True),
        # the diffuse pass on a small odd mesh and on an ordinary one
        dict(name="diffuse_33", kind="diffuse", edge=33),
        dict(name="diffuse_128", kind="diffuse", edge=128),
    ]


def draw(rng):
    logu = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(("step", "step", "step", "surrogate", "batch", "segments", "smooth", "diffuse"))
    if kind == "step":
        edge = logu(20, 160)
        return dict(kind="step", edge=edge, nsrc=logu(1, 400), mesh=rng.choice(("tanh", "tanh", "neutral", "ionized")),
                    sigma=round(rng.uniform(0.3, 1.5), 3), clustered=rng.random() < 0.5,
                    mode=rng.choice(("f32", "f32", "f64")) if edge <= 80 else "f32", overlap=rng.choice((0, 0, 4, 16)))
    if kind == "surrogate":
        return dict(kind="surrogate", edge=logu(20, 110), nsrc=logu(2, 200), mesh=rng.choice(("ionized", "tanh")),
                    sigma=round(rng.uniform(0.3, 1.5), 3), clustered=rng.random() < 0.5)
    if kind == "batch":
        emin = rng.randint(16, 48)
        return dict(kind="batch", nprob=rng.randint(2, 8), emin=emin, emax=rng.randint(emin, 96), smax=logu(8, 300),
                    sigma=round(rng.uniform(0.5, 1.5), 3))
    if kind == "segments":
        return dict(kind="segments", edge=logu(10, 200), nray=logu(1000, 800_000),
                    precision=rng.choice(("kahan", "reference")), sigma=round(rng.uniform(0.3, 1.5), 3))
    if kind == "smooth":
        return dict(kind="smooth", edge=logu(3, 280), isolated=rng.random() < 0.6)
    return dict(kind="diffuse", edge=logu(8, 128))


# ------------------------------------------------------------------ inputs
def _gen(seed, what=0):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + 7919 * what + 1)


def _uniform(g, lo, hi, shape):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64) * (hi - lo) + lo


def _lognormal(edge, sigma, g):
    """Lognormal density of mean 1 with a P(k) ~ k^-3 Gaussian field."""
    if sigma == 0.0:
        return torch.ones(edge ** 3, dtype=torch.float64, device="cuda")
    fk = torch.fft.rfftn(torch.randn((edge,) * 3, generator=g, device="cuda", dtype=torch.float64))
    k = torch.fft.fftfreq(edge, device="cuda", dtype=torch.float64)
    kz = torch.fft.rfftfreq(edge, device="cuda", dtype=torch.float64)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    fk *= k2 ** -0.75
    fk[0, 0, 0] = 0.0
    f = torch.fft.irfftn(fk, s=(edge,) * 3).reshape(-1)
    rho = torch.exp(sigma * f / f.std())
    return rho / rho.mean()


def _ionised_fraction(edge, pos, rate):
    """Largest over the sources of a smoothed top-hat of Stromgren-like radius."""
    x = torch.full((edge,) * 3, 1e-5, dtype=torch.float64, device="cuda")
    c = (torch.arange(edge, device="cuda", dtype=torch.float64) + 0.5) / edge
    for p, n in zip(pos.astype(np.float64), rate):
        R = 0.02 * (n / 1e49) ** (1.0 / 3.0)
        lo = [max(0, int((v - 2.5 * R) * edge)) for v in p]
        hi = [min(edge, int((v + 2.5 * R) * edge) + 2) for v in p]
        s = [slice(a, b) for a, b in zip(lo, hi)]
        r2 = ((c[s[0]] - p[0]) ** 2)[:, None, None] + ((c[s[1]] - p[1]) ** 2)[None, :, None] \
            + ((c[s[2]] - p[2]) ** 2)[None, None, :]
        sub = x[s[0], s[1], s[2]]
        torch.maximum(sub, 0.5 * (1.0 - torch.tanh((r2.sqrt() - R) * (4.0 / R))), out=sub)
    return x.clamp_(1e-5, 0.99).reshape(-1)


def _spectra(rate):
    """Photon rates per frequency bin of blackbodies (nsrc x 256)."""
    edges = 10.0 ** (np.arange(257) * (1.5 / 256))
    u, w = np.polynomial.legendre.leggauss(8)
    mid, half = 0.5 * (edges[1:] + edges[:-1]), 0.5 * np.diff(edges)
    v = mid[:, None] + half[:, None] * u
    counts = ((v * v / np.expm1(H_NUL / (1.38066e-16 * TEMP) * v)) * w).sum(1) * half
    return rate[:, None] * (counts / counts.sum())


def _inputs(case, seed):
    """Fields (float32, flat, z fastest) and sources of one problem."""
    g = _gen(seed)
    edge, ns = case["edge"], case["nsrc"]
    if case["clustered"]:
        centres = _uniform(g, 0.1, 0.9, (32, 3))
        which = torch.randint(0, 32, (ns,), generator=g, device="cuda")
        pos = centres[which] + 0.05 * torch.randn((ns, 3), generator=g, device="cuda", dtype=torch.float64)
    else:
        pos = _uniform(g, 0.0, 1.0, (ns, 3))
    pos = pos.clamp(1e-4, 1.0 - 1e-4).float().cpu().numpy()
    rate = (10.0 ** _uniform(g, 49.0, 51.0, (ns,))).cpu().numpy()
    n = edge ** 3
    dens = _lognormal(edge, case["sigma"], g)
    if case["mesh"] == "tanh":
        x = _ionised_fraction(edge, pos, rate)
        fHI, fHeI, fHeII = 1.0 - x, 1.0 - x, x
    elif case["mesh"] == "neutral":
        x, y = _uniform(g, 1e-4, 1e-2, (n,)), _uniform(g, 1e-4, 1e-2, (n,))
        fHI, fHeI, fHeII = 1.0 - x, 1.0 - y, y
    else:
        fHI, fHeI, fHeII = (1e-4 * 10.0 ** _uniform(g, -0.5, 0.5, (n,)) for _ in range(3))
    return [t.float() for t in (dens, fHI, fHeI, fHeII)], pos, rate


def _workload(case, seed):
    fields, pos, rate = _inputs(case, seed)
    n = len(rate)
    return Workload("case", case["edge"], *(t.cpu().numpy() for t in fields), src_pos=pos, src_rate=rate,
                    src_type=np.zeros(n, np.int32), src_param=np.full(n, TEMP, np.float32), theta=THETA,
                    lunit=LUNIT, denstonh=DENSTONH, src_spectra=_spectra(rate))


def _batch_problems(case, seed):
    """The problems of a batch: the largest and the smallest mesh, the rest between."""
    r = np.random.default_rng(seed)
    out = []
    for i in range(case["nprob"]):
        f = 1.0 - i / max(1, case["nprob"] - 1)
        edge = int(round(case["emin"] + f * (case["emax"] - case["emin"])))
        out.append((dict(edge=edge, nsrc=int(r.integers(4, max(5, case["smax"]))), mesh="tanh", sigma=case["sigma"],
                         clustered=False), 1000 * seed + i))
    return out


def _segment_inputs(case, seed):
    g = _gen(seed)
    dens = _lognormal(case["edge"], case["sigma"], g)
    fr = [_uniform(g, 1e-4, 1.0, (case["edge"] ** 3,)) for _ in range(3)]
    ray = torch.arange(case["nray"], device="cuda")
    ray = torch.repeat_interleave(ray, 1 + ray % 3)
    pos = _uniform(g, 1e-5, 1.0 - 1e-5, (ray.numel(), 6)).float()
    return [t.float() for t in (dens, *fr)], pos, ray


def _smooth_inputs(case, seed):
    """Rates of 1e-12 /s and heating of 1e-24 erg/s, a decade of spread from cell to cell."""
    g = _gen(seed)
    n = case["edge"] ** 3
    f = 10.0 ** torch.randn((6, n), generator=g, device="cuda", dtype=torch.float32)
    return f * torch.tensor([1e-12] * 3 + [1e-24] * 3, device="cuda")[:, None]


def _diffuse_inputs(case, seed):
    """dens, fHI, fHII, fHeI, fHeII, fHeIII, felec, uene of a partly ionised mesh at 2e3 to 5e4 K."""
    g = _gen(seed)
    n = case["edge"] ** 3
    dens = _lognormal(case["edge"], 0.8, g)
    x = _uniform(g, 1e-4, 1.0, (n,)) ** 2
    y = -torch.log(_uniform(g, 1e-6, 1.0, (3, n)))
    y = y / y.sum(0)
    felec = x + HE * (y[1] + 2.0 * y[2])
    uene = 10.0 ** _uniform(g, -0.6, 0.8, (n,))
    return torch.stack([dens, 1.0 - x, x, y[0], y[1], y[2], felec, uene]).float()


# --------------------------------------------------------- prepare and run
def prepare(case, seed):
    kind = case["kind"]
    grid = unit_box_grid(case["edge"], LUNIT, DENSTONH) if "edge" in case else None
    lib = L.load()
    if kind in ("step", "surrogate"):
        pb = Problem(_workload(case, seed))
        st = dict(case=case, pb=pb, buffers=pb.alloc_group_buffers(),
                  rates=torch.zeros(6 * pb.ncell, dtype=torch.float32, device="cuda"))
        if kind == "surrogate":
            pb.set_blackbody()
            st.update(net=Surrogate.from_file(), work=pb.surrogate_work())
        return st
    if kind == "batch":
        b = Batch([_workload(c, s) for c, s in _batch_problems(case, seed)])
        b.configure(mode=1, parts=4)
        return dict(case=case, batch=b)
    if kind == "segments":
        fields, pos, ray = _segment_inputs(case, seed)
        packed = torch.empty(8 * case["edge"] ** 3, dtype=torch.float32, device="cuda")
        L.check(lib.argot_b200_pack_fields(C.byref(grid), *(f.data_ptr() for f in fields), packed.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream), "pack_fields")
        return dict(case=case, lib=lib, grid=grid, packed=packed, pos=pos, ray=ray,
                    seg=torch.empty((ray.numel(), 3), dtype=torch.float32, device="cuda"),
                    out=torch.empty((case["nray"], 3), dtype=torch.float32, device="cuda"))
    if kind == "smooth":
        f = _smooth_inputs(case, seed)
        return dict(case=case, lib=lib, grid=grid, f=f, out=torch.empty_like(f))
    return dict(case=case, grid=grid, f=_diffuse_inputs(case, seed), art=Diffuse(),
                rates=torch.zeros(6 * case["edge"] ** 3, dtype=torch.float32, device="cuda"))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        pb = state["pb"]
        pb.pack()
        if case["mode"] == "f64":
            state["rates"].zero_()  # these rates are added to what is there
            r = pb.run(L.PRECISION_REFERENCE, L.RATE_EXACT_F64, state["rates"], state["buffers"],
                       overlap=case["overlap"])
        else:
            r = pb.run(L.PRECISION_KAHAN, L.RATE_EXACT_F32, state["rates"], state["buffers"], overlap=case["overlap"])
        return list(r.view(6, -1))
    if kind == "surrogate":
        pb, (rays, tau), g = state["pb"], state["buffers"], state["pb"].groups[0]
        pb.pack()
        pb.emit(g, rays)
        pb.march(g, rays, tau)
        pb.rates_surrogate(g, rays, tau, state["rates"], state["net"], work=state["work"])
        return list(state["rates"].view(6, -1))
    if kind == "batch":
        state["batch"].graph_launch()
        return [list(r.view(6, -1)) for r in state["batch"].rates]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "segments":
        prec = L.PRECISION_KAHAN if case["precision"] == "kahan" else L.PRECISION_REFERENCE
        lib, nseg = state["lib"], state["ray"].numel()
        L.check(lib.argot_b200_march_segments(C.byref(state["grid"]), state["packed"].data_ptr(), nseg,
                                              state["pos"].data_ptr(), state["seg"].data_ptr(), prec, stream),
                "march_segments")
        L.check(lib.argot_b200_stitch(nseg, state["ray"].data_ptr(), state["seg"].data_ptr(), case["nray"],
                                      state["out"].data_ptr(), stream), "stitch")
        return [state["seg"], state["out"]]
    if kind == "smooth":
        L.check(state["lib"].argot_b200_smooth_rates(C.byref(state["grid"]), state["f"].data_ptr(),
                                                     state["out"].data_ptr(), int(case["isolated"]), stream), "smooth")
        return list(state["out"])
    state["rates"].zero_()  # the diffuse rates are added to what is there
    state["art"].rates(state["grid"], UENETOK, state["f"], state["rates"])
    return list(state["rates"].view(6, -1))


# -------------------------------------------------------- cost and accuracy
def _rays_per_cell(nsrc):
    """Light rays per target cell at opening angle 0.5 (measured 15 at 16 sources, 190 at 4096)."""
    return nsrc / (1.0 + nsrc / (23.0 * math.log(2.0 + nsrc)))


def work(case):
    """Each input read and each output written once.  Operations: a crossing three multiply-adds and
    ten of geometry, a frequency bin the two optical depths, an attenuation, six sums (45), a diffuse
    step three attenuations and intensities (60)."""
    kind = case["kind"]
    if kind == "batch":
        parts = [work(dict(c, kind="step", mode="f32")) for c, _ in _batch_problems(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = case["edge"] ** 3
    if kind in ("step", "surrogate"):
        rays = n * _rays_per_cell(case["nsrc"])
        return {"bytes": 40.0 * n + 2060.0 * case["nsrc"], "flops": rays * (0.55 * case["edge"] * 16.0 + 256.0 * 45.0)}
    if kind == "segments":
        return {"bytes": 12.0 * n + case["nray"] * (2 * (24 + 8 + 12) + 12.0),
                "flops": 2.0 * case["nray"] * case["edge"] * 16.0}
    if kind == "smooth":
        return {"bytes": 48.0 * n, "flops": 6.0 * 28.0 * n}
    return {"bytes": 4.0 * (8 + 12) * n, "flops": 768.0 * 1.9 * n * 60.0}


def tolerance(case):
    kind = case["kind"]
    if kind == "smooth" or (kind == "segments" and case["precision"] == "reference"):
        return "exact"  # defined operation by operation
    if kind == "surrogate":
        return {"rel": 1e-5, "max": 1e-4}  # up to 2.7e-5 off in a cell; rays near the error budget may change sides
    if kind == "segments":
        return {"rel": 2e-6, "max": 2e-5}
    if kind == "diffuse":
        return {"rel": 2e-5, "max": 5e-4}  # float32 positions along the rays: up to 4.4e-6 off in norm
    return {"rel": 4e-6, "max": 4e-5}


# ------------------------------------------------------- float64 references
def _tables():
    """Frequencies (float32 values) and the cross sections of HI, HeI, HeII (256 x 3, float32 values)."""
    v = 10.0 ** ((np.arange(256) + 0.5) * (1.5 / 256))
    cs = np.array([[_sigma(s, x) for s in range(3)] for x in v]).astype(np.float32).astype(np.float64)
    return v.astype(np.float32).astype(np.float64), cs


def _sigma(s, v):
    if v < THR[s]:
        return 0.0
    if s == 1:
        return 7.83e-18 * (1.66 * (v / THR[1]) ** -2.05 - 0.66 * (v / THR[1]) ** -3.05)
    z4 = (1.0, 0.0, 64.0)[s]  # 256 / 4 for the hydrogenic ion
    e = math.sqrt(v / THR[s] - 1.0)
    return 6.3e-18 * z4 / v ** 4 * math.exp(4.0 - 4.0 * math.atan(e) / e) / (1.0 - math.exp(-2.0 * math.pi / e))


def _products(fields):
    d, a, b, c = (f.double() for f in fields)
    return torch.stack([d * a, HE * d * b, HE * d * c], 1)


def _march(edge, n3, start, end):
    """Columns (code units) along segments, float64."""
    d = end - start
    length = d.square().sum(1).sqrt()
    i = (start * edge).floor().clamp(0, edge - 1).long()
    up = (d > 0).long()
    inf = torch.full_like(d, math.inf)
    move = d != 0
    nxt = torch.where(move, ((i + up) / edge - start) / d, inf)
    gap = torch.where(move, 1.0 / (edge * d.abs()), inf)
    sgn, t = 2 * up - 1, torch.zeros_like(length)
    out = torch.zeros((len(d), 3), dtype=torch.float64, device=d.device)
    while True:
        m = nxt.min(1).values
        to = m.clamp(max=1.0)
        c = i.clamp(0, edge - 1)
        out += ((to - t) * length)[:, None] * n3[(c[:, 0] * edge + c[:, 1]) * edge + c[:, 2]]
        t = to
        go = m < 1.0
        if not bool(go.any()):
            return out
        hit = (nxt == m[:, None]) & go[:, None]
        i = i + sgn * hit
        nxt = torch.where(hit, nxt + gap, nxt)


def _emitters(pos, spec):
    """The oct-tree: nodes in preorder (centre, side, sources, first child or sources, subtree end)."""
    ip = (pos.astype(np.float32).astype(np.float64) * 2 ** 21).astype(np.int64)
    key = np.zeros(len(pos), np.uint64)
    for b in range(21):
        for a in range(3):
            key |= (((ip[:, a] >> b) & 1) << (3 * b + 2 - a)).astype(np.uint64)
    order = np.argsort(key, kind="stable")
    lum = spec.sum(1)
    nodes = []

    def add(ids, depth):
        me = len(nodes)
        w = lum[ids]
        nodes.append(dict(c=((pos[ids].astype(np.float64) * w[:, None]).sum(0) / w.sum()).astype(np.float32),
                          side=np.float32(2.0 ** -depth), ids=ids, kids=len(ids) > 1 and depth < 21,
                          spec=spec[ids].sum(0)))
        if nodes[me]["kids"]:
            digit = (key[ids] >> np.uint64(60 - 3 * depth)) & np.uint64(7)
            for c in range(8):
                if (digit == c).any():
                    add(ids[digit == c], depth + 1)
        nodes[me]["end"] = len(nodes)

    add(order, 0)
    return nodes


def _rays(edge, pos, spec):
    """(emitter positions, spectra, per ray its emitter and target cell)"""
    nodes = _emitters(pos, spec)
    n = edge ** 3
    side = float(np.float32(1.0) / np.float32(edge))
    c1 = ((torch.arange(edge, device="cuda", dtype=torch.float64) + 0.5) * side).float()
    cells = torch.arange(n, device="cuda", dtype=torch.int32)
    blocked = torch.zeros(n, dtype=torch.int32, device="cuda")
    th2 = np.float32(THETA) * np.float32(THETA)
    em, tg = [], []
    v = 0
    while v < len(nodes):
        nd = nodes[v]
        sq = [(c1 - float(x)) for x in nd["c"]]
        sq = [x * x for x in sq]
        r2 = ((sq[0][:, None, None] + sq[1][None, :, None]) + sq[2][None, None, :]).reshape(-1)
        act = blocked <= v
        acc = act & (r2 * float(th2) > float(nd["side"] * nd["side"]))
        opn = act & ~acc
        em.append(v)
        tg.append(cells[acc])
        nxt = nd["end"]
        if bool(opn.any()):
            if nd["kids"]:
                blocked[acc] = nd["end"]
                nxt = v + 1
            else:
                for s in nd["ids"]:
                    em.append(len(nodes) + int(s))
                    tg.append(cells[opn])
        v = nxt
    epos = np.concatenate([np.stack([d["c"] for d in nodes]), pos]).astype(np.float64)
    espec = np.concatenate([np.stack([d["spec"] for d in nodes]), spec])
    ray_e = torch.repeat_interleave(torch.tensor(em, device="cuda"), torch.tensor([len(t) for t in tg], device="cuda"))
    return torch.from_numpy(epos).cuda(), torch.from_numpy(espec).cuda(), ray_e, torch.cat(tg).long()


def _step_exact(case, seed):
    edge = case["edge"]
    if edge ** 3 * _rays_per_cell(case["nsrc"]) > 2.0e8:
        return None
    fields, pos, rate = _inputs(case, seed)
    n3 = _products(fields)
    epos, espec, ray_e, ray_c = _rays(edge, pos, _spectra(rate))
    nu, cs = _tables()
    thr = np.array(THR)
    w6 = torch.from_numpy(np.concatenate([cs, cs * np.maximum(nu[:, None] - thr, 0.0) * H_NUL], 1)).cuda()
    cst = torch.from_numpy(cs).cuda().t().contiguous()
    side = float(np.float32(1.0) / np.float32(edge))
    out = torch.zeros((edge ** 3, 6), dtype=torch.float64, device="cuda")
    for a in range(0, len(ray_e), 1 << 22):
        e, c = ray_e[a:a + (1 << 22)], ray_c[a:a + (1 << 22)]
        ijk = torch.stack([c // (edge * edge), (c // edge) % edge, c % edge], 1)
        end = ((ijk + 0.5) * side)
        col = _march(edge, n3, epos[e], end)
        d = end - epos[e]
        r = d.square().sum(1).sqrt()
        delta = (r[:, None] * side / d.abs().clamp(min=1e-300)).min(1).values
        ok = r > 0
        nt = n3[c]
        D = nt * (delta * LUNIT * DENSTONH)[:, None]
        N = col * (LUNIT * DENSTONH) - 0.5 * D
        P = torch.where(ok, 1.0 / (4.0 * math.pi * LUNIT ** 2 * (r * r + delta * delta / 12.0)), torch.zeros_like(r))
        P6 = (P[:, None] * (nt > 0)).repeat(1, 2)
        for b in range(0, len(e), 1 << 18):
            s = slice(b, b + (1 << 18))
            x = D[s] @ cst
            w = espec[e[s]] * torch.exp(-(N[s] @ cst)) * torch.where(x > 0, -torch.expm1(-x) / x, torch.ones_like(x))
            out.index_add_(0, c[s], torch.where(ok[s, None], P6[s] * (w @ w6), torch.zeros_like(P6[s])))
    return list(out.t())


def _smooth_exact(case, seed):
    e = case["edge"]
    f = _smooth_inputs(case, seed).double().view(6, e, e, e)
    out = 29.0 * f
    idx = torch.arange(e, device="cuda")
    near = [(idx + k).clamp(0, e - 1) if case["isolated"] else (idx + k) % e for k in (-1, 0, 1)]
    for a in near:
        for b in near:
            for c in near:
                out += f[:, a][:, :, b][:, :, :, c]
    return list((out / 56.0).reshape(6, -1))


def _directions():
    """768 HEALPix directions and the face each one enters through (axis, from the low side)."""
    ns, out = 8, []
    c45 = math.cos(math.pi / 4)
    for ring in range(1, 4 * ns):
        i = min(ring, 4 * ns - ring, ns)
        if ring < ns:
            z = 1.0 - ring * ring / (3.0 * ns * ns)
        elif ring <= 3 * ns:
            z = (2 * ns - ring) * 2.0 / (3.0 * ns)
        else:
            z = -1.0 + i * i / (3.0 * ns * ns)
        for k in range(1, 4 * i + 1):
            half = 0.5 if ring < ns or ring > 3 * ns or (ring + ns) % 2 == 0 else 1.0
            phi, th = (k - half) * math.pi / (2.0 * i), math.acos(z)
            cp, sp, tt = math.cos(phi), math.sin(phi), math.tan(th)
            flat = 0 if abs(cp) >= c45 else 1
            lead = 1.0 / abs((cp, sp)[flat])
            axis, low = (2, 1 if tt >= 0 else 0) if abs(tt) <= lead else (flat, int((cp, sp)[flat] >= 0.0))
            o = [math.sin(th) * cp, math.sin(th) * sp, math.cos(th)]
            out.append(([math.copysign(max(abs(v), 1e-31), v) for v in o], axis, low))
    return out


def _recombination(t):
    """Ground-state recombination coefficients of HII, HeII, HeIII (case A minus case B)."""
    l, tev = torch.log(t * 8.61623e-5), t * 8.61623e-5
    p = torch.full_like(t, -3.071135243196595e-9)
    for c in (-1.856767039775261e-8, 5.755614137575758e-7, 4.989108920299513e-6, -0.00001421502914054107,
              -0.0003212605213188796, -0.002380861877349834, -0.02026044731984691, -0.7241125657826851,
              -28.61303380689232):
        p = p * l + c
    hyd_b = lambda lam, a: a * lam ** 1.5 / (1.0 + (lam / 2.740) ** 0.407) ** 2.242  # noqa: E731
    low = 3.92e-13 / tev ** 0.6353
    hot = 1.54e-9 * (1.0 + 0.3 / torch.exp(8.099328789667 / tev)) / (torch.exp(40.49664394833662 / tev) * tev ** 1.5)
    he2_a = torch.where(tev > 0.8, hot + low, low)
    he2_b = torch.where(t > 500.3, 1.26e-14 * (2.0 * 285335.0 / t) ** 0.75,
                        (1.12e-10 - 2.1e-11 * torch.log10(t)) / t.sqrt())
    he3_a = 3.36e-10 / t.sqrt() / (t / 1e3) ** 0.2 / (1.0 + (t / 1e6) ** 0.7)
    return (torch.exp(p) - hyd_b(2.0 * 157807.0 / t, 2.753e-14), he2_a - he2_b,
            he3_a - hyd_b(2.0 * 631515.0 / t, 1.3765e-14))


def _step_factors():
    """4 pi sigma / (h nu) and its heating moment over the first 0.063 above each edge, trapezoidal,
    summed in float32 as the table is defined."""
    out = []
    for s, nul in enumerate((3.2885e15, 5.9483e15, 1.3154e16)):
        f = [np.float32(0.0), np.float32(0.0)]
        for k in range(64):
            v = [THR[s] + (k + j) * (0.0632353 / 64) for j in (0, 1)]
            v = [x + 1e-7 if x == THR[s] else x for x in v]
            c = [4.0 * math.pi * _sigma(s, x) / (6.626e-27 * (x * nul)) for x in v]
            h = (0.0 if k == 0 else c[0] * (v[0] - THR[s]), c[0] * (v[1] - THR[s]))
            f = [np.float32(float(f[0]) + 0.5 * sum(c)), np.float32(float(f[1]) + 0.5 * sum(h))]
        out.append((float(f[0] / np.float32(64)), float(np.float32(float(f[1]) / (64 / (6.626e-27 * nul))))))
    return out


def _diffuse_exact(case, seed):
    e = case["edge"]
    n = e ** 3
    d, h1, h2, e1, e2, e3, fe, u = _diffuse_inputs(case, seed).double()
    t = (u * UENETOK / ((1.0 + fe) * 0.755 + 0.25 * 0.245)).clamp(min=1.0)
    nh = d * DENSTONH
    ne = nh * (h2 + HE * (e2 + 2.0 * e3))
    cs = [float(np.float32(_sigma(s, THR[s] + 1e-7))) for s in range(3)]
    k1, k2, k3 = cs[0] * h1 * nh, cs[1] * HE * e1 * nh, cs[2] * HE * e2 * nh
    ab = torch.stack([k1, k1 * 1.9529766579e-01 + k2, k1 * 1.9513732355e-02 + k2 * 2.6858709594e-01 + k3], 1) + 1e-31
    ion = (h2 * nh, HE * e2 * nh, HE * e3 * nh)
    S = torch.stack([r * ne * x * (13.6 * w * 1.6022e-12 / (4.0 * math.pi))
                     for r, x, w in zip(_recombination(t), ion, THR)], 1) / ab
    offs = torch.tensor([0.521212345, 0.508512345, 0.468287655], dtype=torch.float64, device="cuda")
    mean = torch.zeros((n, 3), dtype=torch.float64, device="cuda")  # sum over directions of absorbed / chord
    dirs = _directions()
    q = torch.arange(e * e, device="cuda")
    per = max(1, (1 << 20) // (e * e))
    for a0 in range(0, len(dirs), per):
        part = dirs[a0:a0 + per]
        na = len(part)
        o = torch.tensor([x[0] for x in part], device="cuda").float().double()
        axis = torch.tensor([x[1] for x in part], device="cuda")
        low = torch.tensor([x[2] for x in part], device="cuda")
        ijk = torch.zeros((na, e * e, 3), dtype=torch.long, device="cuda")
        side = torch.tensor([[1, 2], [0, 2], [0, 1]], device="cuda")[axis]
        ijk.scatter_(2, side[:, :1, None].expand(-1, e * e, 1), (q // e)[None, :, None].expand(na, -1, 1))
        ijk.scatter_(2, side[:, 1:, None].expand(-1, e * e, 1), (q % e)[None, :, None].expand(na, -1, 1))
        face = axis[:, None, None].expand(-1, e * e, 1)
        ijk.scatter_(2, face, torch.where(low > 0, 0, e - 1)[:, None, None].expand(-1, e * e, 1))
        i = ijk.reshape(-1, 3)
        og = o.repeat_interleave(e * e, 0)
        ax = axis.repeat_interleave(e * e)
        base = torch.arange(na, device="cuda").repeat_interleave(e * e) * n
        up = (og > 0).long()
        frac = torch.where(torch.arange(3, device="cuda")[None, :] == ax[:, None], (1 - up).double(), offs[None, :])
        gap = 1.0 / (e * og.abs())
        nxt = torch.where(up > 0, 1.0 - frac, frac) * gap
        I = torch.zeros((len(i), 3), dtype=torch.float64, device="cuda")
        s = torch.zeros(len(i), dtype=torch.float64, device="cuda")
        acc = torch.zeros((na * n, 4), dtype=torch.float64, device="cuda")
        while len(i):
            m = nxt.min(1).values
            chord = (m - s) * LUNIT
            cell = (i[:, 0] * e + i[:, 1]) * e + i[:, 2]
            tau = ab[cell] * chord[:, None]
            em = -torch.expm1(-tau)
            acc.index_add_(0, base + cell, torch.cat([I * em, chord[:, None]], 1))
            I = I * torch.exp(-tau) + S[cell] * em
            s = m
            hit = nxt == m[:, None]
            i = i + (2 * up - 1) * hit
            nxt = torch.where(hit, nxt + gap, nxt)
            out = (i < 0) | (i >= e)
            on = ~out.gather(1, ax[:, None])[:, 0]
            I = torch.where(out.any(1, keepdim=True), torch.zeros_like(I), I)  # wrapped rays start afresh
            i = i % e
            if not bool(on.all()):
                i, og, ax, base, up, gap, nxt, I, s = (x[on] for x in (i, og, ax, base, up, gap, nxt, I, s))
        acc = acc.view(na, n, 4)
        mean += (acc[:, :, :3] / acc[:, :, 3:]).sum(0)
    J = mean / ab + len(dirs) * S
    st = _step_factors()
    hi = J[:, 0] + 1.128855608262e-01 * J[:, 1] + 5.288790581895e-03 * J[:, 2]
    hh = J[:, 0] + 3.1154224364e+00 * J[:, 1] + 5.2452188546e-01 * J[:, 2]
    g = (hi * st[0][0], (J[:, 1] + 1.2404369898e-01 * J[:, 2]) * st[1][0], J[:, 2] * st[2][0],
         hh * st[0][1], (J[:, 1] + 8.7872474963e+00 * J[:, 2]) * st[1][1], J[:, 2] * st[2][1])
    return [x / len(dirs) for x in g]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "surrogate"):
        return _step_exact(case, seed)
    if kind == "batch":
        return [_step_exact(c, s) or [None] * 6 for c, s in _batch_problems(case, seed)]
    if kind == "segments":
        fields, pos, ray = _segment_inputs(case, seed)
        pos = pos.double()
        seg = _march(case["edge"], _products(fields), pos[:, :3], pos[:, 3:])
        out = torch.zeros((case["nray"], 3), dtype=torch.float64, device="cuda")
        return [seg, out.index_add_(0, ray, seg)]
    return _smooth_exact(case, seed) if kind == "smooth" else _diffuse_exact(case, seed)
