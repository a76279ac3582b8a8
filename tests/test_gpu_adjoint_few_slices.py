"""The adjoint of volumes of one to five slices, whose warps take no more lanes than
that along z, and of volumes with enough blocks of 32 columns (smaller ones take 8): <A x, y> = <x, A' y> for every detector row's y.  All terms are
positive, both sides have the same weights, and each sum's relative error is at
most a rounding of 2^-24 for each product and addition of its terms."""
import numpy as np
import pytest

from conftest import dev, geo, host

pytestmark = pytest.mark.gpu


# (columns of a block: 256 for one slice, 128 for two, 64 for three and four)
@pytest.mark.parametrize("nz,nx,ny", [(1, 257, 5), (1, 31, 40), (2, 129, 33), (3, 65, 20), (4, 64, 31),
                                      (5, 33, 32), (64, 65, 70), (65, 66, 77)])
def test_adjoint_of_shallow_volumes_row_by_row(ctx, torch_cuda, nz, nx, ny):
    torch = torch_cuda
    na, nb = 77, 2 * nz + 1
    g = geo(nx=nx, ny=ny, nz=nz, na=na, nb=nb, SO=300.0, SD=450.0, da=5.3, db=0.9, bi=0.21)
    a = [g[k] for k in ("SO", "SD", "da", "na", "ai", "db", "nb", "bi", "nx", "ny", "nz")]
    rng = np.random.default_rng(nz)
    x = rng.random((nz, ny, nx), dtype=np.float32) + np.float32(0.5)
    y = rng.random((nb, na), dtype=np.float32) + np.float32(0.5)
    proj = torch.zeros((nb, na), device="cuda")
    back = torch.full((nz, ny, nx), 7.0, device="cuda")
    # a ray has at most 3 x 2 voxels in a slab, a voxel 3 columns x nb rows of two axes;
    # two roundings a term, and y's and x's products here in FP64
    tol = 2.0 ** -23 * (6 * max(nx, ny) + 6 * nb)
    for angle in (0.3, 0.7853982, 1.5, 3.9):
        ctx.host_projection(proj, dev(torch, x), angle, *a)
        ctx.synchronize()
        ax = host(proj).astype(np.float64)
        for r in range(nb) if nz <= 5 else (0, 1, nb // 3, nb // 2, nb - 1):
            yr = np.zeros_like(y)
            yr[r] = y[r]
            ctx.host_backprojection_adjoint(back, dev(torch, yr), angle, *a)
            ctx.synchronize()
            lhs, rhs = float((ax * yr).sum()), float((x.astype(np.float64) * host(back)).sum())
            assert lhs >= 0 and abs(lhs - rhs) <= tol * lhs, (angle, r, lhs, rhs)
