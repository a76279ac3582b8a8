"""The warps of volumes of every shape, rows beyond what a grid dimension of eight
rows a block could hold among them.  With no displacement a voxel of the result is
a voxel of the source (exactly: the weights are 0 and 1)."""
import numpy as np
import pytest

from conftest import dev, host

pytestmark = pytest.mark.gpu

SHAPES = [(4, 524289, 1), (1, 524289, 3), (524289, 4, 1), (8, 8, 3000), (33, 7, 5), (12, 40, 9),
          (1, 1, 40), (64, 64, 3)]


@pytest.mark.parametrize("shape", SHAPES)
def test_warps_without_displacement(torch_cuda, shape):
    import mcsart_b200 as m
    torch = torch_cuda
    nx, ny, nz = shape
    img = np.random.default_rng(nx).random((nz, ny, nx), dtype=np.float32)
    # memory position r of a slice is (ix, iy) = (r / ny, r % ny), sampled at (x, y) = (iy, ix)
    r = np.arange(nx * ny)
    want = img[:, np.minimum(r // ny, ny - 1), np.minimum(r % ny, nx - 1)].reshape(img.shape)
    d_img, zero = dev(torch, img), torch.zeros((6, nz, ny, nx), device="cuda")
    out = torch.full((nz, ny, nx), 7.0, device="cuda")
    with m.Context(0, stream=torch.cuda.current_stream().cuda_stream) as ctx:
        ctx.set_interp(m.INTERP_EXACT)
        ctx.host_deform(out, d_img, nx, ny, nz, 0.7, 0.3, *zero)
        ctx.synchronize()
        np.testing.assert_array_equal(host(out), want)
        ctx.host_deform2(out, d_img, nx, ny, nz, 0.7, 0.3, *zero)
        ctx.synchronize()
        np.testing.assert_array_equal(host(out), img)
        out16 = torch.zeros((nz, ny, nx), device="cuda", dtype=torch.bfloat16)
        ctx.deform_ex(out16, d_img, nx, ny, nz, 0.7, 0.3, zero.bfloat16())
        ctx.synchronize()
        np.testing.assert_array_equal(host(out16.float()), host(dev(torch, want).bfloat16().float()))
