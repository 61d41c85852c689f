"""The NumPy restatement of the source oct-tree against the library's host
tree: the same nodes, centres and spectra bit for bit."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.parametrize("make", ["plain", "precision", "one", "two"])
def test_restated_tree_equals_the_host_tree(make):
    from argot_b200 import _lib as L, workload as W
    from argot_b200.pipeline import photon_counts, unit_box_grid
    from oracle.tree import Tree
    wl = {"plain": lambda: W.plain(16, 16, seed=1), "precision": lambda: W.precision(seed=2),
          "one": lambda: W.tiny(16, 1, seed=3), "two": lambda: W.tiny(16, 2, seed=4)}[make]()
    spec = np.ascontiguousarray(W.photon_rates(photon_counts, wl.src_type, wl.src_param, wl.src_rate))
    pos = np.ascontiguousarray(wl.src_pos, np.float32)
    lib, tree = L.load(), C.c_void_p()
    g = unit_box_grid(wl.edge, wl.lunit, wl.denstonh)
    L.check(lib.argot_b200_tree_build(C.byref(g), len(pos), pos.ctypes.data, spec.ctypes.data, float(wl.theta),
                                      C.byref(tree)), "tree_build")
    n = lib.argot_b200_tree_num_emitters(tree)
    p4, s = np.zeros((n, 4), np.float32), np.zeros((n, 256))
    L.check(lib.argot_b200_tree_emitters(tree, p4.ctypes.data, s.ctypes.data), "tree_emitters")
    lib.argot_b200_tree_free(tree)
    got_pos, got_spec = Tree(pos, spec).emitters()
    assert np.array_equal(got_pos, p4[:, :3]) and np.array_equal(got_spec, s)
