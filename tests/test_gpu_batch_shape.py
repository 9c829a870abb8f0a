"""The collision tile shape chosen for a batch's members (mpcd_ctx_collide_shape) is the one the batch's
launches use, before the first step and after captured ones, and leaves the states as every other does."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import modulated_state, poiseuille_params
from tests.test_gpu_f64_batch import _native

pytestmark = pytest.mark.gpu

# (cells, threads) of a block by shape (csrc/cells.cuh)
SHAPES = {0: (32, 128), 1: (64, 256), 2: (128, 256), 3: (256, 512)}


def _collide_blocks(step):
    """step() under the profiler: the (blocks, threads) of its collision launches."""
    import json
    import tempfile

    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        step()
    with tempfile.NamedTemporaryFile(suffix=".json") as f:
        prof.export_chrome_trace(f.name)
        events = json.load(open(f.name))["traceEvents"]
    kernels = [e for e in events if e.get("cat") == "kernel"]
    if not kernels:
        pytest.skip("no kernel trace on this machine")
    return {(e["args"]["grid"][0], e["args"]["block"][0]) for e in kernels if "k_f64_collide" in e["name"]}


def test_batch_uses_its_members_shape():
    native = _native()
    cases = [poiseuille_params(61, 37, 9), poiseuille_params(40, 55, 12)]
    states = [modulated_state(p, 20 + k) for k, p in enumerate(cases)]
    alone = []
    for p, (x, v) in zip(cases, states):
        with native.Context(p) as ctx:
            ctx.set_state(x, v)
            ctx.step(0, 3 * len(SHAPES))
            alone.append(ctx.get_state())
    with native.Batch(cases) as B:
        for i, (x, v) in enumerate(states):
            B.member(i).set_state(x, v)
        step = 0
        for k, (cells, threads) in SHAPES.items():
            for i in range(len(cases)):
                B.member(i).collide_shape(k)
            blocks = sum(-(-p["Nc"] // cells) for p in cases)
            assert _collide_blocks(lambda: B.step(step, 3)) == {(blocks, threads)}, k
            step += 3
        for i, (xa, va) in enumerate(alone):
            xg, vg = B.member(i).get_state()
            assert np.array_equal(xg, xa) and np.array_equal(vg, va), i


@pytest.mark.parametrize("shape", range(7))
def test_states_of_every_shape(shape):
    native = _native()
    cases = [poiseuille_params(61, 37, 30), poiseuille_params(9, 7, 40)]
    states = [modulated_state(p, 20 + k) for k, p in enumerate(cases)]
    with native.Batch(cases) as B:
        for i, (x, v) in enumerate(states):
            B.member(i).set_state(x, v)
            B.member(i).collide_shape(shape)
        B.step(0, 4)
        got = [B.member(i).get_state() for i in range(len(cases))]
    for p, (x, v), (xg, vg) in zip(cases, states, got):
        with native.Context(p) as ctx:
            ctx.set_state(x, v)
            ctx.step(0, 4)
            xa, va = ctx.get_state()
        assert np.array_equal(xg, xa) and np.array_equal(vg, va)
