"""Reading the state into device buffers: written in place where kernels may write the buffer, through
id buckets where the output outgrows the L2 cache (n >= 4,194,304), staged otherwise. Every way
gives the values that the host read gives (positions and velocities are copies: equality)."""
import numpy as np
import pytest

from src_incompressible_openmp_b200.cases import poiseuille_params, uniform_state

pytestmark = pytest.mark.gpu

# the last two around the bucket path's threshold: 4,194,303 particles stay direct; 4,300,023
# leave a ragged last bucket, tile and cell run
SIZES = [("f64", 33, 17, 300), ("f32", 33, 17, 3000), ("fast", 33, 17, 3000), ("f64", 1024, 512, 4194303),
         ("f64", 1021, 421, 4300023), ("fast", 1021, 421, 4300023), ("f32", 1021, 421, 4300023)]


@pytest.mark.parametrize("form,Nx,Ny,n", SIZES)
def test_device_read_equals_host_read(form, Nx, Ny, n):
    import torch

    from src_incompressible_openmp_b200 import native
    if not native.device_available():
        pytest.fail("no sm_100 device: the CUDA path has no CPU fallback")
    p = poiseuille_params(Nx, Ny, 10, n=n, gamma=max(1.0, n / (Nx * Ny)))
    x, v = uniform_state(p, 5)
    with native.Context(p, form=form) as ctx:
        ctx.set_state(x, v)
        ctx.step(0, 2)
        xh, vh = ctx.get_state()
        assert np.isfinite(xh).all() and np.isfinite(vh).all()

        def read(off, want=(True, True)):
            """Into device buffers that start `off` doubles past an allocation's start."""
            buf = torch.full((2, 2 * n + 2), 7.0, dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            ctx.get_state_device(*[b.data_ptr() + 8 * off if w else 0 for b, w in zip(buf, want)])
            got = buf.cpu().numpy()
            assert (got[:, :off] == 7.0).all() and (got[:, 2 * n + off:] == 7.0).all()
            return got[:, off:2 * n + off]

        for off in (0, 1):  # 16-byte aligned and not
            xd, vd = read(off)
            assert np.array_equal(xd, xh) and np.array_equal(vd, vh)
        assert np.array_equal(read(0, (True, False))[0], xh)
        assert np.array_equal(read(0, (False, True))[1], vh)
        # the state is untouched by the reads, and loads back from device buffers (FP32 state is
        # exact in FP64, so its reload is)
        if form != "fast":
            d = torch.from_numpy(np.stack([xh, vh])).cuda()
            torch.cuda.synchronize()
            ctx.set_state_device(d[0].data_ptr(), d[1].data_ptr())
            x2, v2 = ctx.get_state()
            assert np.array_equal(v2, vh)
            assert np.array_equal(x2, xh) if form == "f64" else np.allclose(x2, xh, rtol=0, atol=1e-6)
