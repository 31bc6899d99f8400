"""Native handles are freed before the context they were made on, once each, however Python comes
to drop them: a backend in a garbage cycle with its objects (a script's globals at exit) included.
No GPU: the library is a recorder."""
import ctypes as C
import gc

import pytest

import saddlepoint_b200 as sp
from saddlepoint_b200 import batch


class Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda h: self.calls.append((name, getattr(h, "value", h)))


@pytest.fixture
def lib(monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(sp, "library", lambda: rec)
    return rec


def make_backend(lib, value=1):
    import weakref

    b = object.__new__(sp.CudaBackend)
    b.lib, b.h = lib, C.c_void_p(value)
    b._children = weakref.WeakSet()
    b._live = {}
    return b


def attached(kind, backend, value):
    h = object.__new__(kind)
    h._attach(backend, C.c_void_p(value))
    return h


KINDS = [(sp.Solver, "sp_solver_free"), (sp.Problem, "sp_problem_free"), (sp.Vector, "sp_vec_free"),
         (batch._BatchHandle, "sp_batch_free"), (batch._ServerHandle, "sp_server_destroy")]


def check(lib, objects):
    assert lib.calls[-1] == ("sp_ctx_destroy", 1) and len(lib.calls) == objects + 1
    assert len(set(lib.calls)) == len(lib.calls)


@pytest.mark.parametrize("backend_first", [True, False])
def test_a_garbage_cycle_frees_the_objects_before_the_context(backend_first, lib):
    for _ in range(4):
        lib.calls.clear()
        ring = []
        if backend_first:
            ring.append(make_backend(lib))
        backend = ring[0] if ring else make_backend(lib)
        for k, (kind, _) in enumerate(KINDS):
            ring.append(attached(kind, backend, 10 + k))
        if not backend_first:
            ring.append(backend)
        for x in ring:
            x.ring = ring  # a cycle through every object
        del x, backend, ring
        gc.collect()
        check(lib, len(KINDS))
        assert sorted(lib.calls[:-1]) == sorted((free, 10 + k) for k, (_, free) in enumerate(KINDS))


def test_closing_the_backend_first_leaves_the_objects_without_a_handle(lib):
    backend = make_backend(lib)
    objects = [attached(kind, backend, 10 + k) for k, (kind, _) in enumerate(KINDS)]
    backend.close()
    check(lib, len(KINDS))
    assert all(o.h is None for o in objects)
    for o in objects:
        o.close()
    backend.close()
    check(lib, len(KINDS))


def test_a_handle_that_was_closed_is_not_freed_again(lib):
    backend = make_backend(lib)
    a, b = attached(sp.Vector, backend, 10), attached(sp.Vector, backend, 11)
    a.close()
    a.close()
    c = attached(sp.Vector, backend, 10)  # the address again
    backend.close()
    assert sorted(lib.calls[:-1]) == [("sp_vec_free", 10), ("sp_vec_free", 10), ("sp_vec_free", 11)]
    assert lib.calls[-1] == ("sp_ctx_destroy", 1) and b.h is None and c.h is None
