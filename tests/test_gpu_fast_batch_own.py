"""A fast batch whose replicas have stepped on their own, unequal numbers of times, before its first step and
between steps: their bins lie differently and their collision tiles have been tuned one by one, and every
replica still equals itself stepped alone, bit for bit."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import poiseuille_params, uniform_state
from tests.test_gpu_fast_batch import _native

pytestmark = pytest.mark.gpu

CASES = [(8, 28, 15, {}), (23, 11, 4, {}), (13, 20, 8, {}),
         (8, 34, 10, dict(boundary_left="bounceback", boundary_right="specular", Utop=0.05))]
# per replica the steps taken alone, as (step0, nsteps)
SCHEDULES = {
    "before the first": [[(0, 1)], [(0, 2)], [(0, 1)], [(0, 2)]],
    "several": [[(0, 1), (1, 1)], [(0, 3), (5, 1)], [(0, 2), (2, 3)], [(0, 4)]],
    "one replica": [[], [], [(0, 1)], []],
}


@pytest.mark.parametrize("metrics", [False, True])
@pytest.mark.parametrize("name", sorted(SCHEDULES))
def test_unequal_steps_alone(name, metrics):
    native = _native()
    cases = [poiseuille_params(Nx, Ny, ppc, **over) for Nx, Ny, ppc, over in CASES]
    states = [uniform_state(p, 82 + k) for k, p in enumerate(cases)]
    own = SCHEDULES[name]
    want = []
    for p, (x, v), alone in zip(cases, states, own):
        with native.Context(p, form="fast") as ctx:
            ctx.set_state(x, v)
            for s in alone:
                ctx.step(*s, metrics=metrics)
            ctx.step(6, 3)
            ctx.step(9, len(alone))
            ctx.step(20, 4)
            want.append(ctx.get_state())
    with native.Batch(cases, form="fast") as B:
        for i, (x, v) in enumerate(states):
            B.member(i).set_state(x, v)
            for s in own[i]:
                B.member(i).step(*s, metrics=metrics)
        B.step(6, 3)
        for i in range(len(cases)):
            B.member(i).step(9, len(own[i]))
        B.step(20, 4)
        for i, (xa, va) in enumerate(want):
            xg, vg = B.member(i).get_state()
            assert np.array_equal(xg, xa) and np.array_equal(vg, va), i
