"""The stencil launchers on slices of every shape: narrow ones, where a row or a
column is a voxel or a few, both sides of host_add2's tiled form, and a volume
whose index comes to the end of 31 bits."""
import numpy as np
import pytest

from conftest import dev, host

pytestmark = pytest.mark.gpu

SHAPES = [(1, 70, 9), (70, 1, 9), (1, 1, 300), (5, 3, 401), (15, 33, 20), (33, 15, 20), (16, 16, 5), (56, 52, 55),
          (35, 37, 33), (1025, 2, 1)]


def _fwd(a, axis):
    d = np.zeros_like(a)
    n = a.shape[axis]
    i, j = [slice(None)] * 3, [slice(None)] * 3
    i[axis], j[axis] = slice(0, n - 1), slice(1, n)
    d[tuple(i)] = a[tuple(j)] - a[tuple(i)]
    return d


@pytest.mark.parametrize("shape", SHAPES)
def test_stencils_match_their_formulas(ctx, torch_cuda, shape):
    """diff, initial2 and multiple round as NumPy's float32 operations (bits must
    agree); add2 adds with one rounding, checked against float64 to an ulp."""
    torch = torch_cuda
    nx, ny, nz = shape
    rng = np.random.default_rng(nx * ny)
    a, b, c = (rng.random((nz, ny, nx), dtype=np.float32) for _ in range(3))
    out = torch.zeros((nz, ny, nx), device="cuda")
    d = {1: _fwd(c, 2), 2: _fwd(c, 1), 3: _fwd(c, 0)}
    w = np.float32(0.7)
    ctx.host_initial2(out, nx, ny, nz, dev(torch, c), 0.3, 0.2)
    ctx.synchronize()
    np.testing.assert_array_equal(host(out), ((d[1] + d[2]) + d[3]) * (np.float32(0.3) + np.float32(0.2)))
    # img is read at iy + ix*ny within a slice
    t = b.reshape(nz, nx, ny).transpose(0, 2, 1)
    for ind in (1, 2, 3):
        ctx.host_diff(out, dev(torch, c), nx, ny, nz, ind)
        ctx.synchronize()
        ref = np.zeros_like(c)
        ax = 3 - ind
        n = c.shape[ax]
        if n > 2:
            i, j = [slice(None)] * 3, [slice(None)] * 3
            i[ax], j[ax] = slice(1, n - 1), slice(0, n - 2)
            ref[tuple(i)] = c[tuple(i)] - c[tuple(j)]
        np.testing.assert_array_equal(host(out), ref)
        m = dev(torch, a)
        ctx.host_multiple(m, nx, ny, nz, dev(torch, c), 0.7, ind)
        ctx.synchronize()
        np.testing.assert_array_equal(host(m), a * (w * d[ind]))
        s = dev(torch, a)
        ctx.host_add2(s, dev(torch, b), nx, ny, nz, dev(torch, c), 0.7, ind)
        ctx.synchronize()
        ref = a.astype(np.float64) + (t * w).astype(np.float64) * d[ind]
        assert np.all(np.abs(host(s) - ref) <= 2.0 ** -24 * np.abs(ref) + 1e-45)


@pytest.mark.parametrize("shape", [(1, 2 ** 31 - 1, 1), (1, 1, 2 ** 31 - 1)])
def test_the_largest_index(ctx, torch_cuda, shape):
    """Two arrays of 2^31 - 1 voxels: no coordinate or index wraps."""
    torch = torch_cuda
    n = 2 ** 31 - 1
    img = torch.arange(n, device="cuda", dtype=torch.int32).bitwise_and_(0xFFFF).to(torch.float32)
    out = torch.full((n,), 7.0, device="cuda")
    ctx.host_diff(out, img, *shape, 1 + int(np.argmax(shape)))
    ctx.synchronize()
    assert out[0] == 0 and out[n - 1] == 0
    step = 1 << 28
    for i in range(1, n - 1, step):
        j = min(i + step, n - 1)
        assert torch.equal(out[i:j], img[i:j] - img[i - 1:j - 1])
    del img, out
    torch.cuda.empty_cache()
