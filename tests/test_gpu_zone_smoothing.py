"""A 391x58 channel at 19 particles per cell (replica 30 of the ensemble family of seed 20) whose
second step has a zone that is sensitive to the order in which its sparse cells see their
neighbours: steps against the oracle, positions and moves exact."""
import math

import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import ensemble_family

pytestmark = pytest.mark.gpu
REL = 1e-9


def _native():
    from src_incompressible_openmp_b200 import native
    if not native.device_available():
        pytest.fail("no sm_100 device: the CUDA path has no CPU fallback")
    return native


@pytest.mark.parametrize("seed", [1030, 2030])
def test_steps_of_a_sensitive_replica(oracle, seed):
    import torch
    native = _native()
    p = ensemble_family(64, 20)[30][0]
    g = torch.Generator(device="cuda:0")
    g.manual_seed(seed)
    x = torch.rand((p["n"], 2), generator=g, device="cuda:0", dtype=torch.float64)
    x[:, 0] *= p["Lx"]
    x[:, 1] *= p["Ly"]
    v = torch.randn((p["n"], 2), generator=g, device="cuda:0", dtype=torch.float64)
    v *= math.sqrt(p["kBT"])
    v -= v.mean(dim=0)
    xo, vo = x.cpu().numpy().reshape(-1).copy(), v.cpu().numpy().reshape(-1).copy()
    with native.Context(p) as ctx:
        for s in range(1, 4):
            ctx.set_state(xo, vo)
            m = ctx.step(s - 1, 1, metrics=True)
            xg, vg = ctx.get_state()
            xo, vo, mo = oracle.step(p, xo, vo, s)
            assert np.array_equal(xg, xo), s
            assert np.max(np.abs(vg - vo) / np.maximum(1.0, np.abs(vo))) <= REL, s
            for ph in ("base", "shifted"):
                for k in ("nParticlesMovedDense", "nParticlesMovedSparse"):
                    assert m[ph][k] == mo[ph][k], (s, ph, k)
