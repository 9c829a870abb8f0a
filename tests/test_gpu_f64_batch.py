"""The plain batch with one launch per phase: replicas of uneven size (fewer than a block, more than
one block of every launch, walls all round, no particles, an unequal number of steps taken on
their own) equal the same replicas stepped alone, bit for bit; an error of one replica is
reported."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import modulated_state, poiseuille_params, uniform_state

pytestmark = pytest.mark.gpu

BOX = dict(boundary_left="specular", boundary_right="bounceback", Utop=0.1)
SETS = {
    # 25 zones in all: one zone per block; 2 to 170 cells of a last block
    "small": [(7, 6, 9, {}), (33, 17, 12, {}), (16, 16, 1, BOX)],
    # above 592 zones: zones in step, eight to a block, none of the zone counts a multiple of 8
    "large": [(161, 73, 5, {}), (256, 256, 3, dict(bodyForceX=5e-3)), (97, 41, 14, BOX), (12, 10, 20, {})],
}


def _native():
    from src_incompressible_openmp_b200 import native
    if not native.device_available():
        pytest.fail("no sm_100 device: the CUDA path has no CPU fallback")
    return native


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("name", sorted(SETS))
def test_batch_equals_alone(name, graphs):
    native = _native()
    cases = [poiseuille_params(Nx, Ny, ppc, **over) for Nx, Ny, ppc, over in SETS[name]]
    cases.append(poiseuille_params(20, 10, 10, n=0))
    states = [modulated_state(p, 80 + k) if p["n"] else (np.zeros(0), np.zeros(0)) for k, p in enumerate(cases)]
    alone = []
    for p, (x, v) in zip(cases, states):
        with native.Context(p) as ctx:
            ctx.set_state(x, v)
            ctx.step(0, 7)
            alone.append(ctx.get_state())
    with native.Batch(cases) as B:
        for i, (x, v) in enumerate(states):
            B.member(i).set_state(x, v)
            B.member(i).set_graphs(graphs)
        B.step(0, 1)
        B.step(1, 3)
        # a step of every member on its own, then the last ones together
        for i in range(len(cases)):
            B.member(i).step(4, 1)
        B.step(5, 2)
        for i, (xa, va) in enumerate(alone):
            xg, vg = B.member(i).get_state()
            assert np.array_equal(xg, xa) and np.array_equal(vg, va), i


def test_batch_reports_a_members_error():
    native = _native()
    good = poiseuille_params(20, 12, 10)
    bad = poiseuille_params(20, 12, 10, boundary_top="sticky")
    with native.Batch([good, bad]) as B:
        for i, p in enumerate((good, bad)):
            B.member(i).set_state(*uniform_state(p, 90 + i))
        with pytest.raises(native.MpcdError) as e:
            B.step(0, 3)
        assert e.value.code == 3 and "boundary_top" in str(e.value)
