"""Zone passes whose thresholds have integer tables (dense cells decided on integers, donors ranked
without their noise draws where the ranking is certain) and those next to the tables' limits:
bit-identical to the oracle in positions and velocities, with its moved counts."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import modulated_state, poiseuille_params, uniform_state

pytestmark = pytest.mark.gpu

CASES = [
    ("channel", 41, 23, 10, {}),
    ("integer thresholds", 30, 20, 8, dict(coef=0.0)),  # low = high = gamma
    ("wide band", 30, 20, 12, dict(coef=0.37, highMode="1+coef", lowMode="1+coef")),
    ("low override", 30, 20, 9, dict(lowThrBulkOverride=8.999999999999998)),
    ("empty-cell floors inside the band", 26, 22, 9, dict(lowThrFloor=9.25, highThrFloor=9.75)),
    ("one particle per cell", 40, 30, 1, {}),  # low threshold 0.9: the general routines
    ("tables' upper limit", 14, 12, 115, {}),  # high threshold 126.5
    ("beyond the limit", 14, 12, 116, {}),     # 127.6: the general routines
    ("odd tiles", 31, 29, 10, dict(zoneTileNx=3, zoneTileNy=7)),
    ("two-cell tiles", 17, 9, 10, dict(zoneTileNx=2, zoneTileNy=2)),
    ("tile next to the period", 13, 12, 10, dict(boundary_bottom="periodic", boundary_top="periodic", zoneTileNx=11,
                                                zoneTileNy=10)),
    ("walls all round", 23, 21, 10, dict(boundary_left="specular", boundary_right="bounceback")),
]


@pytest.mark.parametrize("name,Nx,Ny,ppc,over", CASES, ids=[c[0].replace(" ", "_") for c in CASES])
def test_zone_pass_equals_oracle(oracle, name, Nx, Ny, ppc, over):
    from src_incompressible_openmp_b200 import native
    if not native.device_available():
        pytest.fail("no sm_100 device: the CUDA path has no CPU fallback")
    p = poiseuille_params(Nx, Ny, ppc, **over)
    states = [uniform_state(p, 71), modulated_state(p, 72, mode="checker"), modulated_state(p, 73, amp=0.95)]
    with native.Context(p) as ctx:
        for k, (x, v) in enumerate(states):
            ctx.set_state(x, v)
            for mode, seed in (("base", 88172645463325252 + 10007 * k), ("shifted", 88172645463325252 + 4099 + 10007 * k)):
                xin, vin = ctx.get_state()
                mg = ctx.zone_pass(mode, seed)
                xo, vo, mo = oracle.zone_pass(p, xin, vin, mode, seed)
                xg, vg = ctx.get_state()
                assert np.array_equal(xg, xo), (k, mode)
                assert np.array_equal(vg, vo), (k, mode)
                for key in ("nParticlesMovedDense", "nParticlesMovedSparse", "corrMaxDU"):
                    assert mg[key] == mo[key], (k, mode, key)
