"""The pool of page-locked result arrays: blocks that are in use are not handed out again, what is dropped is
reused, what does not fit its bound is an ordinary array. On the CPU with a library that only counts."""
import gc
import sys

import numpy as np
import pytest

from tissueorigami_b200 import capi, hostmem, mesh

MB = 1 << 20


class _Lib:
    def __init__(self):
        self.live = {}

    def tf_host_register(self, handle, p, n):
        assert handle == "ctx" and p % 4096 == 0 and p not in self.live
        self.live[p] = n
        return 0

    def tf_host_unregister(self, p):
        del self.live[p]
        return 0


@pytest.mark.parametrize("doubles", [MB // 8 - 1, MB // 8, MB // 8 + 1, 5 * MB // 8 + 3, 40 * MB // 8])
def test_pool_reuses_only_what_was_dropped(doubles):
    pool, lib = hostmem._Pool(), _Lib()
    a = pool.take(lib, "ctx", (doubles,))
    if 8 * doubles < hostmem.MIN_BYTES:
        assert a is None
        return
    b = pool.take(lib, "ctx", (doubles,))
    a[:], b[:] = 1.0, 2.0
    assert (a == 1.0).all() and (b == 2.0).all() and len(lib.live) == 2
    view, where = a[5:9], a.ctypes.data
    del a
    gc.collect()
    c = pool.take(lib, "ctx", (doubles,))  # the view still holds the first block
    assert c.ctypes.data not in (where, b.ctypes.data) and (view == 1.0).all()
    del view
    gc.collect()
    d = pool.take(lib, "ctx", (doubles,))
    assert d.ctypes.data == where and len(lib.live) == 3


def test_pool_is_bounded():
    pool, lib = hostmem._Pool(), _Lib()
    held = [pool.take(lib, "ctx", (30 * MB // 8,)) for _ in range(8)]
    assert all(h is not None for h in held) and sum(lib.live.values()) <= hostmem.LIMIT
    assert pool.take(lib, "ctx", (30 * MB // 8,)) is None
    assert pool.take(lib, "ctx", (hostmem.LIMIT // 8 + 1,)) is None
    del held
    gc.collect()
    assert sum(lib.live.values()) <= hostmem.KEEP
    other = pool.take(lib, "ctx", (250 * MB // 8,))  # gives the kept blocks back
    assert other is not None and sum(lib.live.values()) <= hostmem.LIMIT


@pytest.mark.parametrize("what", ["mmap", "madvise"])
def test_a_refused_mapping_is_no_error(monkeypatch, what):
    """Without a mapping the result is an ordinary array, without huge pages the block has small ones."""
    real = hostmem.mmap.mmap

    class Mapping(real):
        def madvise(self, *args):
            raise OSError(22, "Invalid argument")

    def refuse(*args, **kw):
        raise OSError(12, "Cannot allocate memory")

    monkeypatch.setattr(hostmem.mmap, "mmap", refuse if what == "mmap" else Mapping)
    pool, lib = hostmem._Pool(), _Lib()
    a = pool.take(lib, "ctx", (MB // 8,))
    assert (a is None) == (what == "mmap") and len(lib.live) == (what == "madvise")
    assert pool._bytes == sum(lib.live.values())


def test_arrays_dropped_while_another_is_taken():
    """The garbage collector may drop arrays between any two lines of take() on the same thread: no block is
    handed out twice, none is lost, and the bound holds."""
    pool, lib = hostmem._Pool(), _Lib()

    def garbage(mb):
        a = pool.take(lib, "ctx", (mb * MB // 8,))
        cycle = [a]
        cycle.append(cycle)

    lines = [0]

    def trace(frame, event, arg):
        if frame.f_code.co_filename != hostmem.__file__ or frame.f_code.co_name in ("_give", "_reset"):
            return None
        if event == "line":
            lines[0] += 1
            if lines[0] == at:
                gc.collect()
        return trace

    gc.disable()
    gc.freeze()  # collections look at what follows only
    try:
        for at in range(1, 60):
            for sizes in ([1, 2, 3], [3, 2, 1], [70, 1, 1]):
                held = [pool.take(lib, "ctx", (MB // 8,)) for _ in range(2)]
                del held  # two kept blocks
                for mb in sizes:
                    garbage(mb)
                lines[0] = 0
                sys.settrace(trace)
                try:
                    held = [pool.take(lib, "ctx", (mb * MB // 8,)) for mb in (1, 2, 1)]
                finally:
                    sys.settrace(None)
                spans = sorted((h.ctypes.data, h.nbytes) for h in held)
                assert all(p + n <= q for (p, n), (q, _) in zip(spans, spans[1:]))
                assert all(p in lib.live for p, _ in spans)
                del held
                gc.collect()
                assert sum(lib.live.values()) == pool._bytes <= hostmem.KEEP
    finally:
        gc.unfreeze()
        gc.enable()


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(11, 11), (41, 40)])
def test_results_equal_those_in_ordinary_arrays(nx, ny):
    """J of 0.7 and 9 MB, assembled in the coloured scatter's fixed order."""
    from tissueorigami_b200.newton import NewtonRaphsonSolver

    t = mesh.large_slab(nx=nx, ny=ny)
    with NewtonRaphsonSolver.from_tissue(t, scatter=2) as s:
        first = s.assemble(t.x, t.x, t.dt)
        keep = first[1].copy()
        second = s.assemble(t.x * 1.001, t.x, t.dt)
        np.testing.assert_array_equal(first[1], keep)
        assert np.abs(second[1] - first[1]).max() > 0
        x = np.ascontiguousarray(t.x, dtype=np.float64).reshape(-1)
        g, vals = np.empty(x.shape), np.empty(keep.shape)
        capi.check(s._L.tf_assemble(s._h, capi.dptr(x), capi.dptr(x), t.dt, capi.dptr(g), capi.dptr(vals)), "tf_assemble", s._h)
        np.testing.assert_array_equal(vals, keep)
    np.testing.assert_array_equal(first[1], keep)  # the arrays outlive the context
