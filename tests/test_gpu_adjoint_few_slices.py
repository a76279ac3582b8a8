"""The adjoint of volumes of one to five slices, whose warps take no more lanes than
that along z, against the FP64 oracle with the bound of the parity tests (1e-5
relative L2)."""
import numpy as np
import pytest

from conftest import dev, geo, host, rel_l2

pytestmark = pytest.mark.gpu


# (columns of a block: 256 for one slice, 128 for two, 64 for three and four)
@pytest.mark.parametrize("nz,nx,ny", [(1, 257, 5), (1, 31, 40), (2, 129, 33), (3, 65, 20), (4, 64, 31),
                                      (5, 33, 32)])
def test_adjoint_of_shallow_volumes(ctx, torch_cuda, oracle, nz, nx, ny):
    torch = torch_cuda
    g = geo(nx=nx, ny=ny, nz=nz, na=77, nb=2 * nz + 1, SO=300.0, SD=450.0, da=5.3, db=0.9, bi=0.21)
    p = np.random.default_rng(nz).random((g["nb"], 77), dtype=np.float32)
    out = torch.full((nz, ny, nx), 7.0, device="cuda")
    for a in (0.3, 0.7853982, 1.5, 3.9):
        ctx.host_backprojection_adjoint(out, dev(torch, p), a, g["SO"], g["SD"], g["da"], 77, g["ai"],
                                        g["db"], g["nb"], g["bi"], nx, ny, nz)
        ctx.synchronize()
        o = oracle.backprojection_adjoint(p, a, g)
        assert np.linalg.norm(o) > 0 and rel_l2(host(out), o) <= 1e-5, (a, rel_l2(host(out), o))
