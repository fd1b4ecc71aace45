"""The Python mirror's buffers: an array of the host mapping stays readable after free(), and the memory goes back with the last
such array.  Against a stand-in for the library's allocator: no GPU."""
import ctypes as C
import gc

import numpy as np
import pytest

from rknpu2_matmul_open_b200 import capi, rmsnorm


class _Handle:
    handle = 1
    ctx = None


@pytest.fixture
def library(monkeypatch):
    class Library:
        blocks, freed = {}, []

        def rk_npu_mem_alloc(self, domain, size, flags, out):
            block = (C.c_uint8 * size)()
            mem = out._obj
            mem.handle, mem.size, mem.vaddr = len(self.blocks) + 1, size, C.addressof(block)
            self.blocks[mem.handle] = block
            return capi.RK_NPU_OK

        def rk_npu_mem_free(self, ctx, out):
            mem = out._obj
            self.freed.append(mem.handle)
            C.memset(C.byref(mem), 0, C.sizeof(mem))
            return capi.RK_NPU_OK

    lib = Library()
    lib.blocks, lib.freed = {}, []
    monkeypatch.setattr(capi, "load", lambda: lib)
    return lib


def _domain():
    dom, ctx = _Handle(), _Handle()
    dom.ctx = ctx
    return dom


def test_memory_goes_back_at_once_without_arrays(library):
    b = rmsnorm.Buffer(_domain(), 64)
    b.array()[:] = 7                            # a passing array
    gc.collect()
    assert b.free() == capi.RK_NPU_OK and library.freed == [1] and b.mem.handle == 0
    assert b.free() == capi.RK_NPU_OK and library.freed == [1]


def test_an_array_outlives_its_buffer(library):
    b = rmsnorm.Buffer(_domain(), 64)
    rows = b.array().reshape(4, 8)[1:]
    rows[:] = 5
    assert b.free() == capi.RK_NPU_OK and library.freed == [] and b.mem.handle == 0
    again = rows[0]
    del b, rows
    gc.collect()
    assert library.freed == [] and np.all(again == 5)
    del again
    gc.collect()
    assert library.freed == [1]


def test_a_buffer_that_was_never_freed_keeps_its_memory(library):
    b = rmsnorm.Buffer(_domain(), 64)
    view = b.array()
    del b, view
    gc.collect()
    assert library.freed == []
