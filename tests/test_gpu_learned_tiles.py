"""The training kernel's gradient at the edges of its 128-row tiles and of the four groups that share a
tile's hidden units, against the float64 oracle with the kernel's BF16 operands (the tolerances of
test_learned.py: FP32 accumulation order, 1e-4 of the largest entry)."""
import numpy as np
import pytest

from tests.test_learned import MO, _native, _rand_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [2, 31, 127, 128, 129, 257, 512])
def test_gradient_at_tile_edges(rows):
    native = _native()
    X, Y, p = _rand_case(rows, 200 + rows)
    g, loss = native.learned_grad(X, Y, p)
    loss_o, g_o = MO.loss_grad_tc(X, Y, p)
    assert abs(loss - loss_o) <= 1e-5 * loss_o
    assert np.max(np.abs(g - g_o)) <= 1e-4 * np.max(np.abs(g_o))
