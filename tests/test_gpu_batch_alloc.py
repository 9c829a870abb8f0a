"""A device allocation that fails during a batch's first step: the call reports it, the members' states stay
as they were, and the next call makes what is missing and steps. The failure is a fake of the allocation call
on the host (mpcd_device_malloc), each allocation of the first step failing in turn."""
import ctypes as C

import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import poiseuille_params, uniform_state
from tests.test_gpu_f64_batch import _native

pytestmark = pytest.mark.gpu

MALLOC = C.CFUNCTYPE(C.c_int, C.POINTER(C.c_void_p), C.c_size_t)
OUT_OF_MEMORY = 2  # cudaErrorMemoryAllocation


class FailingMalloc:
    """The library's device allocations, counted; number `fail` (from 0) reports that memory is short."""

    def __init__(self, lib, fail=None):
        self.slot = C.c_void_p.in_dll(lib, "mpcd_device_malloc")
        self.real = self.slot.value
        self.count = 0
        real = MALLOC(self.real)

        def call(p, size):
            k, self.count = self.count, self.count + 1
            return OUT_OF_MEMORY if k == fail else real(p, size)

        self.fake = MALLOC(call)

    def __enter__(self):
        self.slot.value = C.cast(self.fake, C.c_void_p).value
        return self

    def __exit__(self, *a):
        self.slot.value = self.real


@pytest.mark.parametrize("form", ["f64", "fast"])
def test_first_step_after_a_failed_one(form):
    native = _native()
    cases = [poiseuille_params(20, 10, 20), poiseuille_params(13, 17, 20)]
    states = [uniform_state(p, 40 + k) for k, p in enumerate(cases)]

    def filled():
        B = native.Batch(cases, form=form)
        for i, (x, v) in enumerate(states):
            B.member(i).set_state(x, v)
        return B

    def read(B):
        return [B.member(i).get_state() for i in range(len(cases))]

    with filled() as B:
        with FailingMalloc(native.lib()) as m:
            B.step(0, 3)
        want = read(B)
    assert m.count > 0
    for fail in range(m.count):
        with filled() as B:
            before = read(B)
            with FailingMalloc(native.lib(), fail), pytest.raises(native.MpcdError):
                B.step(0, 3)
            for (xa, va), (xb, vb) in zip(before, read(B)):
                assert np.array_equal(xa, xb) and np.array_equal(va, vb)
            B.step(0, 3)
            for (xa, va), (xb, vb) in zip(want, read(B)):
                assert np.array_equal(xa, xb) and np.array_equal(va, vb), fail
