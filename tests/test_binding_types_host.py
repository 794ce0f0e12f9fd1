"""Argument types of the single calls in the Python binding, on the CPU: only
vectors and tables are unwrapped, any other object with a pointer is refused
before the C call (here a stand-in for the library that counts its calls)."""
import ctypes
import types

import pytest

import vkhel_gb300 as vk

CALLS = {
    "elemfma": ("vvv", (3, 17)), "elemfma_canonical": ("vvv", (3, 17)), "elemmul": ("vvv", (17,)),
    "elemmod": ("vv", (5, 17)), "elemgtadd": ("vv", (5, 3)), "elemgtsub": ("vv", (5, 3, 17)),
    "forward_transform": ("vvt", ()), "inverse_transform": ("vvt", ()),
}


def _object(cls):
    # no device here: an address stands for the C object, and nothing frees it
    plain = type(cls.__name__, (cls,), {"__del__": lambda self: None})
    x = plain.__new__(plain)
    x.ctx = types.SimpleNamespace(ptr=None)
    x.ptr = 0x1000
    return x


@pytest.fixture
def calls(monkeypatch):
    made = []

    class Stub:
        def __getattr__(self, name):
            sig = next(s for s in vk._SIGNATURES if s[0] == name)

            def record(*args):
                made.append(name)
                return 0

            return ctypes.CFUNCTYPE(sig[1], *sig[2])(record)

    monkeypatch.setattr(vk, "_lib", Stub())
    return made


def _args(kinds):
    return [_object(vk.Vector if k == "v" else vk.NttTables) for k in kinds]


@pytest.mark.parametrize("name", sorted(CALLS))
def test_vectors_and_tables_reach_the_library(calls, name):
    kinds, rest = CALLS[name]
    getattr(vk, name)(*_args(kinds), *rest)
    assert calls[0] == "vkhel_vector_" + name


@pytest.mark.parametrize("wrong", [vk.Batch, vk.ElemBatch, vk.Server])
@pytest.mark.parametrize("name", sorted(CALLS))
def test_other_objects_are_refused(calls, name, wrong):
    kinds, rest = CALLS[name]
    for at in range(len(kinds)):
        args = _args(kinds)
        args[at] = _object(wrong)
        with pytest.raises(ctypes.ArgumentError):
            getattr(vk, name)(*args, *rest)
    assert calls == []
