"""The adjoint gather at the edges of its blocks: 32 columns of one row by 32
slices, or 8 where 32 would leave a quarter of the lanes idle (depth 31, 32 and
64 take the first, the others the second form); one detector row, rows past the
tile of 32 and footprints of several rows and slices.  Against the FP64 oracle's
adjoint with the bound of the adjoint's tests (1e-5 relative L2)."""
import numpy as np
import pytest

from conftest import dev, geo, host, rel_l2

pytestmark = pytest.mark.gpu

# (nx, ny, nz, na, nb, da, db)
SHAPES = [(1, 1, 1, 2, 2, 0.9, 0.8), (31, 33, 8, 33, 1, 0.9, 5.0), (32, 31, 9, 32, 31, 0.9, 0.8),
          (33, 32, 31, 64, 33, 0.7, 1.6), (65, 20, 32, 31, 64, 2.6, 0.4),
          (20, 40, 33, 70, 65, 0.5, 3.1), (24, 24, 64, 40, 97, 0.9, 0.9)]


@pytest.mark.parametrize("shape", SHAPES)
def test_adjoint_at_block_edges_matches_the_oracle(ctx, torch_cuda, oracle, shape):
    torch = torch_cuda
    nx, ny, nz, na, nb, da, db = shape
    # (one voxel: a near source, whose coordinates' rounding is below the bound)
    SO = 90.0 if nx > 1 else 8.0
    g = geo(nx=nx, ny=ny, nz=nz, na=na, nb=nb, SO=SO, SD=1.5 * SO, da=da, db=db, ai=0.37, bi=-0.61)
    p = np.random.default_rng(nz).random((nb, na), dtype=np.float32)
    out = torch.full((nz, ny, nx), 7.0, device="cuda")
    for a in (0.3, 0.7853982, 1.5, 3.9, 5.2):
        ctx.host_backprojection_adjoint(out, dev(torch, p), a, g["SO"], g["SD"], g["da"], na,
                                        g["ai"], g["db"], nb, g["bi"], nx, ny, nz)
        ctx.synchronize()
        o = oracle.backprojection_adjoint(p, a, g)
        assert np.linalg.norm(o) > 0 and rel_l2(host(out), o) <= 1e-5, (a, rel_l2(host(out), o))
