"""Handles are freed once, also when the interpreter is ending and the
modules' names are gone."""
import ctypes as C

import pytest


class _Lib:
    """records what is freed"""

    def __init__(self):
        self.freed = []

    def __getattr__(self, name):
        return lambda h: self.freed.append((name, h.value))


def _bare(cls, **attrs):
    o = cls.__new__(cls)
    for k, v in attrs.items():
        setattr(o, k, v)
    return o


@pytest.mark.parametrize("names_gone", [False, True])
def test_handles_are_freed_once(monkeypatch, names_gone):
    from argot_b200 import batch, diffuse, pipeline, surrogate
    lib = _Lib()
    pb = _bare(pipeline.Problem, lib=lib, _dtree=C.c_void_p(1), _tree=C.c_void_p(2))
    b = _bare(batch.Batch, lib=lib, handle=C.c_void_p(3), problems=[pb])
    s = _bare(surrogate.Surrogate, lib=lib, handle=C.c_void_p(4))
    d = _bare(diffuse.Diffuse, lib=lib, h=C.c_void_p(5))
    if names_gone:
        for m in (batch, diffuse, pipeline, surrogate):
            monkeypatch.setattr(m, "C", None)
    for _ in range(2):
        for o in (b, pb, s, d):
            o.__del__()
    assert sorted(h for _, h in lib.freed) == [1, 2, 3, 4, 5]
