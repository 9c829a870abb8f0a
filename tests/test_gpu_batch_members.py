"""Batches of small replicas that step on their own streams, joined around the zone passes, because a member
has an option that only its own step implements (mean flow kept, one full-domain zone, the learned closure):
each replica equals the replica alone, bit for bit, eager and replayed, also when the members' buffers come to
lie differently, when a batch goes over from one kind of step to the other between calls, and when an option
changes after steps have been captured."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import poiseuille_params, uniform_state
from tests.test_gpu_f64_batch import _native

pytestmark = pytest.mark.gpu

PLAIN = [(24, 16, 9, {}), (17, 33, 6, dict(bodyForceX=4e-3))]
SPECIAL = {
    "keepMeanFlow": (21, 14, 8, dict(keepMeanFlow=True)),
    "single zone": (16, 12, 8, dict(zoneSingleFullDomainMode=True)),
    "learned": (28, 20, 10, {}),
}


def _cases(name):
    return [poiseuille_params(Nx, Ny, ppc, **over) for Nx, Ny, ppc, over in (PLAIN[0], SPECIAL[name], PLAIN[1])]


def _network(native, seed):
    net = native.learned_init(seed)
    net[-1] = 1e-3
    return net


def _check(native, cases, ops, graphs):
    """ops(i): what happens to replica i, as (kind, ...) tuples; steps are taken together."""
    lists = [ops(i) for i in range(len(cases))]
    want = []
    for p, todo in zip(cases, lists):
        seen = []
        with native.Context(p) as ctx:
            ctx.set_graphs(graphs)
            for op in todo:
                _apply(native, ctx, op, seen, ctx.step)
        want.append(seen)
    got = [[] for _ in cases]
    with native.Batch(cases) as B:
        for i in range(len(cases)):
            B.member(i).set_graphs(graphs)
        for turn in zip(*lists):
            if turn[0][0] == "step":
                assert all(op == turn[0] for op in turn)
                B.step(*turn[0][1:])
                continue
            for i, op in enumerate(turn):
                _apply(native, B.member(i), op, got[i], None)
    for i, (a, b) in enumerate(zip(want, got)):
        for k, ((xa, va), (xb, vb)) in enumerate(zip(a, b)):
            assert np.array_equal(xa, xb) and np.array_equal(va, vb), (i, k)


def _apply(native, ctx, op, seen, step):
    if op[0] == "state":
        ctx.set_state(*uniform_state(ctx.params, op[1]))
    elif op[0] == "learned":
        ctx.learned_set(None if op[1] is None else _network(native, op[1]), *op[2:])
    elif op[0] == "read":
        seen.append(ctx.get_state())
    elif op[0] == "step":
        step(*op[1:])


@pytest.mark.parametrize("graphs", [True, False])
@pytest.mark.parametrize("name", sorted(SPECIAL))
def test_replicas_on_their_own_streams(name, graphs):
    native = _native()

    def ops(i):
        special = ("learned", 5, 10.0) if name == "learned" and i == 1 else ("none",)
        return [("state", 30 + i), special, ("step", 0, 1), ("step", 1, 12), ("read",), ("step", 13, 5), ("read",)]

    _check(native, _cases(name), ops, graphs)


@pytest.mark.parametrize("graphs", [True, False])
def test_buffers_that_lie_differently_and_alike_again(graphs):
    """One replica's state is uploaded again after an odd number of steps, later every replica's: the steps
    captured before see the buffers they were captured with."""
    native = _native()

    def ops(i):
        again = ("state", 50) if i == 1 else ("none",)
        return [("state", 30 + i), ("step", 0, 11), again, ("step", 11, 9), ("read",), ("state", 60 + i),
                ("step", 20, 10), ("read",)]

    _check(native, _cases("keepMeanFlow"), ops, graphs)


@pytest.mark.parametrize("graphs", [True, False])
def test_learned_closure_switched_between_calls(graphs):
    """The batch goes over from batched launches to the members' own streams and back."""
    native = _native()

    def ops(i):
        def learned(*a):
            return ("learned", *a) if i == 1 else ("none",)
        return [("state", 30 + i), ("step", 0, 7), learned(5, 10.0), ("step", 7, 11), ("read",), learned(None),
                ("step", 18, 6), ("read",), learned(6, 1e-6), ("step", 24, 12), ("read",)]

    _check(native, _cases("learned"), ops, graphs)


@pytest.mark.parametrize("graphs", [True, False])
def test_learned_closure_switched_under_captured_steps(graphs):
    """A replica with the mean flow kept holds the batch on the members' own streams throughout; the closure
    of another one changes after the batch's steps have been captured."""
    native = _native()

    def ops(i):
        def learned(*a):
            return ("learned", *a) if i == 2 else ("none",)
        return [("state", 30 + i), ("step", 0, 12), learned(5, 10.0), ("step", 12, 12), ("read",), learned(6, 1e-6),
                ("step", 24, 12), ("read",), learned(None), ("step", 36, 10), ("read",)]

    _check(native, _cases("keepMeanFlow"), ops, graphs)
