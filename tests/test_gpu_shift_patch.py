"""A plain step's closure over the patched index of its in-place shifted pass equals a step that
reports metrics, whose shifted pass makes a fresh index, bit for bit: on even, modulated and clumped
states, where the shifted pass moves from none to many particles per cell."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import modulated_state, poiseuille_params, uniform_state

pytestmark = pytest.mark.gpu

BOX = dict(boundary_left="specular", boundary_right="bounceback", Utop=0.1)


def _native():
    from src_incompressible_openmp_b200 import native
    if not native.device_available():
        pytest.fail("no sm_100 device: the CUDA path has no CPU fallback")
    return native


def clumped_state(p, seed):
    """40 % of the particles in a square blob, ten to 25 times as dense as the mean."""
    x, v = uniform_state(p, seed)
    rng = np.random.default_rng(seed)
    x = x.reshape(-1, 2)
    k = int(0.4 * p["n"])
    side = int(np.ceil(np.sqrt(0.4 * p["Nc"] / 25)))
    for i, (L, N) in enumerate(((p["Lx"], p["Nx"]), (p["Ly"], p["Ny"]))):
        x[:k, i] = 0.5 * L + side * (L / N) * (rng.random(k) - 0.5)
    return x.reshape(-1).copy(), v


def columns_state(p, seed):
    """Every particle in the columns whose number is a multiple of 8: most cells empty."""
    x, v = uniform_state(p, seed)
    x = x.reshape(-1, 2)
    a = p["Lx"] / p["Nx"]
    col = np.floor(x[:, 0] / a)
    x[:, 0] = np.minimum((col - col % 8 + (x[:, 0] / a - col)) * a, p["Lx"] * (1 - 1e-12))
    return x.reshape(-1).copy(), v


STATES = dict(uniform=uniform_state, modulated=modulated_state, clumped=clumped_state, columns=columns_state)


@pytest.mark.parametrize("form", ["f64", "f32"])
@pytest.mark.parametrize("state", sorted(STATES))
@pytest.mark.parametrize("Nx, Ny, ppc, over", [(7, 6, 12, {}), (16, 16, 1, BOX), (33, 17, 10, BOX), (70, 41, 5, {}),
                                               (130, 90, 20, {})])
def test_patched_step_equals_step_with_a_fresh_index(form, state, Nx, Ny, ppc, over):
    native = _native()
    p = poiseuille_params(Nx, Ny, ppc, **over)
    x, v = STATES[state](p, 17)
    ends = []
    for metrics in (False, True):
        with native.Context(p, form=form) as ctx:
            ctx.set_state(x, v)
            for s in range(4):  # eager and replayed steps
                ctx.step(s, 1, metrics=metrics)
            ends.append(ctx.get_state())
    assert np.array_equal(ends[0][0], ends[1][0])
    assert np.array_equal(ends[0][1], ends[1][1])
