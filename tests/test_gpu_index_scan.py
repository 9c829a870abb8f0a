"""The cell index at the edges of its scans' tiles (4,096 values; one block up to 65,536): counts,
momenta and their order against sums over the particles in id order."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import poiseuille_params, uniform_state

pytestmark = pytest.mark.gpu


def _native():
    from src_incompressible_openmp_b200 import native
    if not native.device_available():
        pytest.fail("no sm_100 device: the CUDA path has no CPU fallback")
    return native


# 4, 4095, 4096, 4097, 8191, 8193, 65535, 65536, 65537, 65538 and 69632 cells
@pytest.mark.parametrize("Nx, Ny", [(2, 2), (63, 65), (64, 64), (241, 17), (8191, 1), (2731, 3), (257, 255), (256, 256),
                                    (65537, 1), (331, 198), (272, 256)])
def test_sums_in_id_order(Nx, Ny):
    native = _native()
    p = poiseuille_params(Nx, Ny, 3, n=3 * Nx * Ny)
    x, v = uniform_state(p, 5)
    dx, dy = p["Lx"] / Nx, p["Ly"] / Ny
    ix = np.clip(np.floor(x[0::2] / dx), 0, Nx - 1).astype(np.int64)
    iy = np.clip(np.floor(x[1::2] / dy), 0, Ny - 1).astype(np.int64)
    cid = ix * Ny + iy
    # away from the cells' edges, where a quotient's rounding would decide
    for q, a, i in ((x[0::2], dx, ix), (x[1::2], dy, iy)):
        q[:] = (i + 0.001 + 0.998 * (q / a - i)) * a
    with native.Context(p) as ctx:
        ctx.set_state(x, v)
        f = ctx.cell_fields(3.0)
    assert np.array_equal(f["N"], np.bincount(cid, minlength=Nx * Ny))
    assert np.array_equal(f["Px"], np.bincount(cid, weights=v[0::2], minlength=Nx * Ny))
    assert np.array_equal(f["Py"], np.bincount(cid, weights=v[1::2], minlength=Nx * Ny))


# entries per cell around the rank sort's group sizes (8, 16, 24 and 32 entries, 128 keys of a warp),
# in neighbouring cells and far apart
COUNTS = [0, 1, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33, 63, 64, 65, 127, 128, 129, 257, 700]


@pytest.mark.parametrize("spread", [1, 5, 11])
def test_order_within_cells(spread):
    native = _native()
    Nx, Ny = 23, 13
    counts = np.zeros(Nx * Ny, np.int64)
    counts[(np.arange(len(COUNTS)) * spread + 2) % (Nx * Ny)] = COUNTS
    rng = np.random.default_rng(spread)
    cid = rng.permutation(np.repeat(np.arange(Nx * Ny), counts))
    p = poiseuille_params(Nx, Ny, 10, n=len(cid))
    x = np.empty(2 * len(cid))
    x[0::2] = (cid // Ny + rng.uniform(0.01, 0.99, len(cid))) * (p["Lx"] / Nx)
    x[1::2] = (cid % Ny + rng.uniform(0.01, 0.99, len(cid))) * (p["Ly"] / Ny)
    v = rng.standard_normal(2 * len(cid)) * 10.0 ** rng.integers(-6, 7, len(cid)).repeat(2)  # sums depend on the order
    with native.Context(p) as ctx:
        ctx.set_state(x, v)
        f = ctx.cell_fields(3.0)
    assert np.array_equal(f["N"], counts)
    assert np.array_equal(f["Px"], np.bincount(cid, weights=v[0::2], minlength=Nx * Ny))
    assert np.array_equal(f["Py"], np.bincount(cid, weights=v[1::2], minlength=Nx * Ny))
