"""The fast form's integer zone decisions against the FP64 comparisons they replaced: moved particles and
digests of the states recorded with the revision that decided in FP64, over thresholds with and without
fractional parts, densities, walls, and few and many zones."""
import hashlib

import pytest

from src_incompressible_openmp_b200.cases import modulated_state, poiseuille_params
from tests.test_gpu_fast import _native

pytestmark = pytest.mark.gpu

BOX = dict(boundary_left="bounceback", boundary_right="specular", Utop=0.05)
# (Nx, Ny, particles per cell, parameters) -> (dense and sparse moves of the base and the shifted pass of the
# first step, the state after four steps)
GOLDEN = {
    "few zones": ((947, 214, 10, 18), "585b59d09e5288ab"),
    "odd sizes": ((801, 298, 21, 11), "cfe257229bc05d8f"),
    "dense": ((437, 103, 115, 23), "4779cb75625f9962"),
    "equal fractions": ((599, 281, 84, 10), "a98228961d569d30"),
    "box": ((1179, 271, 9, 2), "ea8654e561f72fd9"),
    "other modes": ((303, 133, 24, 3), "f8355a3d3b399d93"),
    "one per cell": ((500, 0, 38, 0), "bc66051588b36295"),
    "periodic": ((76, 19, 0, 0), "53c8fde102f049ae"),
    "many zones": ((31340, 9217, 416, 391), "48ec1dfba29b243b"),
}


def _run(native, key):
    Nx, Ny, ppc, over = CASES[key]
    p = poiseuille_params(Nx, Ny, ppc, **over)
    with native.Context(p, form="fast") as ctx:
        ctx.set_state(*modulated_state(p, 11))
        row = ctx.step(0, 1, metrics=True)
        ctx.step(1, 3)
        x, v = ctx.get_state()
    moves = tuple(int(row[k][f"nParticlesMoved{w}"]) for k in ("base", "shifted") for w in ("Dense", "Sparse"))
    return moves, hashlib.sha256(x.tobytes() + v.tobytes()).hexdigest()[:16]


CASES = {
    "few zones": (50, 50, 10, {}),
    "odd sizes": (61, 37, 7, dict(coef=0.23, lowThrFloor=3.7, highThrFloor=9.3)),
    "dense": (40, 30, 24, dict(coef=0.05)),
    "equal fractions": (48, 32, 12, dict(coef=0.25, lowThrFloor=9.0, highThrFloor=15.0)),
    "box": (70, 45, 15, dict(coef=0.13, lowThrFloor=0.5, highThrFloor=22.6, **BOX)),
    "other modes": (30, 20, 12, dict(coef=0.37, highMode="1+coef", lowMode="1+coef")),
    "one per cell": (40, 30, 1, {}),
    "periodic": (13, 12, 10, dict(boundary_bottom="periodic", boundary_top="periodic", zoneTileNx=11, zoneTileNy=10)),
    "many zones": (512, 192, 9, dict(coef=0.17)),
}


@pytest.mark.parametrize("key", sorted(CASES))
def test_decisions_of_the_recorded_revision(key):
    assert _run(_native(), key) == GOLDEN[key]
