"""Buffers that a context makes at the first call that needs them: an allocation that fails (a fake of the
allocation call on the host) is reported, and the same call then works as on a fresh context. Each allocation
of the call fails in turn."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import poiseuille_params, uniform_state
from tests.test_gpu_batch_alloc import FailingMalloc
from tests.test_gpu_f64_batch import _native

pytestmark = pytest.mark.gpu


def _learned(native, ctx):
    net = native.learned_init(3)
    net[-1] = 1e-3
    ctx.learned_set(net, 10.0)
    ctx.step(0, 3)
    return ctx.get_state()


def _samples(native, ctx):
    return ctx.learned_samples(0, 2, 7)


def _serial(native, ctx):
    ctx.save_ref()
    ctx.zone_pass_serial("base", 77)
    return ctx.get_state()


def _profile(native, ctx):
    ctx.profile_reset()
    ctx.step(0, 3)
    return (ctx.profile_read()[0],)


def _jobs(native, ctx):
    x, v = ctx.get_state()
    xo, vo = ctx.run_jobs(np.stack([x] * 3), np.stack([v] * 3), 0, 2)
    return np.stack(xo), np.stack(vo)


CALLS = {
    "learned f64": ("f64", _learned), "learned fast": ("fast", _learned), "samples f64": ("f64", _samples),
    "samples fast": ("fast", _samples), "serial": ("f64", _serial), "profile": ("f64", _profile), "jobs": ("f64", _jobs),
}


@pytest.mark.parametrize("name", sorted(CALLS))
def test_call_after_a_failed_allocation(name):
    native = _native()
    form, call = CALLS[name]
    p = poiseuille_params(30, 20, 20)
    state = uniform_state(p, 6)

    def fresh():
        ctx = native.Context(p, form=form)
        ctx.set_state(*state)
        return ctx

    with fresh() as ctx, FailingMalloc(native.lib()) as m:
        want = call(native, ctx)
    assert m.count > 0
    for fail in range(m.count):
        with fresh() as ctx:
            with FailingMalloc(native.lib(), fail), pytest.raises(native.MpcdError):
                call(native, ctx)
            ctx.set_state(*state)
            for a, b in zip(want, call(native, ctx)):
                np.testing.assert_array_equal(a, b)
