"""Batched steps out of sequence (a run stepped again from an earlier step, a call of no steps): the rotation
signs kept from one call are those of the step they are used for. Replicas equal the same sequence on
contexts alone, bit for bit."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import poiseuille_params, uniform_state
from tests.test_gpu_f64_batch import _native

pytestmark = pytest.mark.gpu

# (step0, nsteps): the signs of step 3 are made ahead by the first call and wanted by the last one
SEQUENCES = {
    "one step elsewhere": [(0, 3), (10, 1), (2, 1)],
    "no step elsewhere": [(0, 3), (10, 0), (2, 2)],
    "back and on": [(0, 4), (0, 1), (4, 1), (1, 3)],
}


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("name", sorted(SEQUENCES))
def test_batch_out_of_sequence(name, graphs):
    native = _native()
    cases = [poiseuille_params(24, 16, 9), poiseuille_params(17, 33, 6, bodyForceX=4e-3)]
    states = [uniform_state(p, 30 + k) for k, p in enumerate(cases)]
    with native.Batch(cases) as B:
        for i, (x, v) in enumerate(states):
            B.member(i).set_state(x, v)
            B.member(i).set_graphs(graphs)
        for step0, nsteps in SEQUENCES[name]:
            B.step(step0, nsteps)
        got = [B.member(i).get_state() for i in range(len(cases))]
    for p, (x, v), (xg, vg) in zip(cases, states, got):
        with native.Context(p) as ctx:
            ctx.set_state(x, v)
            for step0, nsteps in SEQUENCES[name]:
                ctx.step(step0, nsteps)
            xa, va = ctx.get_state()
        assert np.array_equal(xg, xa) and np.array_equal(vg, va)
