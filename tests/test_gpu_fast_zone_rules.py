"""The fast form's zone decisions on integer threshold tables, over threshold settings, tiles and
boundaries: one, four and eight zones per block give the same state, moved counts included, from
a state whose density is far from even, and no particle is lost."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import modulated_state, poiseuille_params

pytestmark = pytest.mark.gpu

CASES = [
    (41, 23, 10, {}),
    (30, 20, 8, dict(coef=0.0)),
    (30, 20, 12, dict(coef=0.37, highMode="1+coef", lowMode="1+coef")),
    (26, 22, 9, dict(lowThrFloor=9.25, highThrFloor=9.75)),
    (40, 30, 1, {}),
    (31, 29, 10, dict(zoneTileNx=3, zoneTileNy=7)),
    (13, 12, 10, dict(boundary_bottom="periodic", boundary_top="periodic", zoneTileNx=11, zoneTileNy=10)),
    (260, 250, 6, {}),  # 650 zones: eight per block, in launch order
]


@pytest.mark.parametrize("Nx,Ny,ppc,over", CASES)
def test_same_state_for_every_block_width(Nx, Ny, ppc, over, monkeypatch):
    from src_incompressible_openmp_b200 import native
    if not native.device_available():
        pytest.fail("no sm_100 device: the CUDA path has no CPU fallback")
    p = poiseuille_params(Nx, Ny, ppc, **over)
    x, v = modulated_state(p, 61, amp=0.3, mode="siny")
    got = []
    for warps in (None, "4", "8"):
        if warps:
            monkeypatch.setenv("MPCD_FAST_ZONE_WARPS", warps)
        with native.Context(p, form="fast") as ctx:
            ctx.set_state(x, v)
            row = ctx.step(0, 4, metrics=True)
            got.append(ctx.get_state() + (row["base"]["nParticlesMovedDense"], row["base"]["nParticlesMovedSparse"]))
    for g in got[1:]:
        assert np.array_equal(g[0], got[0][0]) and np.array_equal(g[1], got[0][1]) and g[2:] == got[0][2:]
    xg, vg = got[0][0].reshape(-1, 2), got[0][1].reshape(-1, 2)
    assert np.isfinite(xg).all() and np.isfinite(vg).all()
    a = p["a0"]
    cell = np.minimum((xg[:, 0] / a).astype(int), Nx - 1) * Ny + np.minimum((xg[:, 1] / a).astype(int), Ny - 1)
    assert np.bincount(cell, minlength=Nx * Ny).sum() == p["n"]
