"""The partial gradients of a batch's 128-row tiles are added in a fixed order: gradients, losses and trained
networks are the same in every run, and a gradient is the FP32 sum of its tiles' own gradients in that order
(bit for bit: the tiles' scale 2 / (2 rows) differs from the batch's by a power of two, which no rounding of
the chain feels)."""
import numpy as np
import pytest

from tests.test_learned import _native, _rand_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [1, 2, 4, 8, 16])
def test_gradient_is_the_ordered_sum_of_its_tiles(tiles):
    native = _native()
    X, Y, p = _rand_case(128 * tiles, 700 + tiles)
    part = [native.learned_grad(X[q:q + 128], Y[q:q + 128], p)[0][:-1] / np.float32(tiles)
            for q in range(0, 128 * tiles, 128)]
    order = [*range(4, tiles), *range(2, min(tiles, 4)), *range(min(tiles, 2))]
    want = np.zeros_like(part[0])
    for q in order:
        want = want + part[q]
    for _ in range(4):
        g, _ = native.learned_grad(X, Y, p)
        np.testing.assert_array_equal(g[:-1], want)


@pytest.mark.parametrize("rows,batch", [(4096, 512), (3001, 1000), (40000, 40000)])
def test_training_repeats(rows, batch):
    native = _native()
    X, Y, p = _rand_case(rows, rows)
    first = native.learned_train(X, Y, p, epochs=2, batch=batch, seed=3)
    for _ in range(3):
        net, losses = native.learned_train(X, Y, p, epochs=2, batch=batch, seed=3)
        np.testing.assert_array_equal(net, first[0])
        np.testing.assert_array_equal(losses, first[1])
