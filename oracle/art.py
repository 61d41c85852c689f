"""The ART diffuse-radiation pass in float64 (test infrastructure): per-cell
coefficients, the march of every ray of every direction one after another,
and the six rates.  Slow; for meshes of a few thousand rays.

Nothing here is shared with the device path: positions and path lengths are
doubles, the attenuation is expm1.
"""
import numpy as np


def march(n, d, lunit, ab, S, dirs, faces):
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


def coefficients(f, denstonh, uenetok):
    """Absorption [cm^-1] and source functions of the three frequencies
    (calc_rmesh_data.c:33-111, diffuse_chemistry.c:13-103) in float64."""
    dens, hi, hii, hei, heii, heiii, fe, u = f
    he = 0.0811258278
    t = np.maximum(u * uenetok / ((1 + fe) * 0.755 + 0.25 * 0.245), 1.0)
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


def rates(n, d, lunit, denstonh, uenetok, planes, dirs, faces, step6):
    """The pass's six rate planes of a mesh of n cells with sides d, local
    domain = box: eight planes of fields, directions and their start faces,
    the step factors (HI, HeI, HeII; ionisation and heating each)."""
    ab, S = coefficients(planes.astype(np.float64), denstonh, uenetok)
    shape = tuple(n) + (3,)
    J = march(n, d, lunit, ab.reshape(shape), S.reshape(shape), dirs, faces).reshape(-1, 3) / len(faces)
    st = np.asarray(step6, np.float64)
    return np.stack([(J @ [1, 1.128855608262e-01, 5.288790581895e-03]) * st[0], (J @ [0, 1, 1.2404369898e-01]) * st[2],
                     J[:, 2] * st[4], (J @ [1, 3.1154224364e+00, 5.2452188546e-01]) * st[1],
                     (J @ [0, 1, 8.7872474963e+00]) * st[3], J[:, 2] * st[5]])
