"""ARGOT's source oct-tree and its walk restated in NumPy (test
infrastructure): the emitters and, for given target cells, the light rays of
setup_light_ray_tree.c, where the reference's own C is not at hand.

The construction follows setup_light_ray_tree.c:100-239, 465-571: 63-bit
Morton keys, a node split into its non-empty octants while it holds more
than one source, node centres as luminosity-weighted means (sums child by
child; the root's weighted by the first bin), and the walk :341-354 in single
precision: a node is taken when r^2 theta^2 > side^2.
"""
from __future__ import annotations

import numpy as np


def _sum(a):
    """sum over the first axis, one after another"""
    return np.add.accumulate(a, axis=0)[-1]


class Tree:
    """pos (nsrc, 3) float32, spectra (nsrc, 256) float64, in a unit box."""

    def __init__(self, pos, spectra):
        self.pos = np.ascontiguousarray(pos, np.float32)
        self.spectra = np.ascontiguousarray(spectra, np.float64)
        ip = (self.pos.astype(np.float64) * 2.0 ** 21).astype(np.int64).astype(np.uint64)
        key = np.zeros(len(self.pos), np.uint64)
        for bit in range(21):
            for axis in range(3):
                key |= ((ip[:, axis] >> np.uint64(bit)) & np.uint64(1)) << np.uint64(3 * bit + 2 - axis)
        order = np.argsort(key, kind="stable")
        self._lum = _sum(self.spectra.T)
        self.centre, self.side, self.spec, self.ids, self.has_child, self.skip = [], [], [], [], [], []
        w = self.spectra[:, 0]
        root = _sum(self.pos.astype(np.float64) * w[:, None]) / _sum(w)
        self._add(order, 0, root.astype(np.float32), _sum(self.spectra))
        self._split(0, order, key[order], 60)
        self.skip[0] = len(self.ids)
        self.centre, self.spec = np.stack(self.centre), np.stack(self.spec)

    def _add(self, ids, depth, centre, spec):
        self.ids.append(ids)
        self.side.append(np.float32(2.0 ** -depth))
        self.centre.append(centre)
        self.spec.append(spec)
        self.has_child.append(False)
        self.skip.append(0)
        return len(self.ids) - 1

    def _split(self, me, ids, key, level):
        """children of `me` by the key's octant at bit `level`; the node's
        luminosity, spectrum and weighted position sums"""
        octant = (key >> np.uint64(level)) & np.uint64(7)
        lum, spec, cm = 0.0, np.zeros(self.spectra.shape[1]), np.zeros(3)
        for c in range(8):
            mine = octant == c
            if not mine.any():
                continue
            self.has_child[me] = True
            kid = self._add(ids[mine], 21 - level // 3, None, None)
            if mine.sum() > 1 and level > 0:
                m, s, x = self._split(kid, ids[mine], key[mine], level - 3)
                self.centre[kid] = (x / m).astype(np.float32)
            else:
                j = ids[mine]
                m, s = _sum(self._lum[j]), _sum(self.spectra[j])
                x = _sum(self._lum[j][:, None] * self.pos[j])
                self.centre[kid] = (x * (1.0 / m)).astype(np.float32)
            self.spec[kid] = s
            self.skip[kid] = len(self.ids)
            lum, spec, cm = lum + m, spec + s, cm + x
        return lum, spec, cm

    def emitters(self):
        """positions (n, 3) float32 and spectra (n, 256): the nodes, then the
        sources in input order"""
        return np.concatenate([self.centre, self.pos]), np.concatenate([self.spec, self.spectra])

    def rays(self, centres, theta):
        """(cell, emitter) of every ray to the target cells with the given
        centres (n, 3) float32: cell by cell, in the walk's order"""
        th2 = np.float32(theta) * np.float32(theta)
        nn = len(self.ids)
        cells = np.arange(len(centres))
        blocked = np.zeros(len(centres), np.int64)
        cell, emit = [], []
        v = 0
        while v < nn:
            d = centres - self.centre[v]
            r2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2]
            act = blocked <= v
            take = act & (r2 * th2 > self.side[v] * self.side[v])
            opened = act & ~take
            cell.append(cells[take])
            emit.append(np.full(take.sum(), v))
            nxt = self.skip[v]
            if opened.any():
                if len(self.ids[v]) > 1:
                    if self.has_child[v]:
                        blocked[take] = self.skip[v]
                        nxt = v + 1
                else:
                    cell.append(cells[opened])
                    emit.append(np.full(opened.sum(), nn + self.ids[v][0]))
            v = nxt
        cell, emit = np.concatenate(cell), np.concatenate(emit)
        order = np.argsort(cell, kind="stable")
        return cell[order], emit[order]
