"""The adjoint of tall volumes under steep rays, whose rows' axial ratios are rounded
at a large distance from the centre plane: a row's voxels are all found."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,SO,db", [(64001, 30000.0, 0.37), (40000, 22345.6, 0.81), (9001, 5000.0, 1.3)])
def test_steep_rays_of_tall_volumes(ctx, torch_cuda, nz, SO, db):
    """One detector column over 2 x 2 voxel columns: <A x, e_row> = <x, A' e_row>; a
    row has at most 2 slabs x 2 x 3 voxels (two roundings a term, x below 1)."""
    torch = torch_cuda
    nb = 11
    f = np.float32
    bi = float(f(-(nz // 2) * 1.5 / db - 5.3))  # rows near the bottom face
    a = (float(f(SO)), float(f(1.5 * SO)), 1.0, 1, 0.0, float(f(db)), nb, bi, 2, 2, nz)
    img = torch.rand((nz, 2, 2), device="cuda", generator=torch.Generator(device="cuda").manual_seed(nz))
    p, back = torch.zeros((nb, 1), device="cuda"), torch.zeros((nz, 2, 2), device="cuda")
    for angle in (0.3, 1.5, 3.9):
        ctx.host_projection(p, img, angle, *a)
        for r in range(nb):
            e = torch.zeros((nb, 1), device="cuda")
            e[r] = 1.0
            ctx.host_backprojection_adjoint(back, e, angle, *a)
            ctx.synchronize()
            assert abs(float((back.double() * img.double()).sum()) - float(p[r])) <= 24 * 2.0 ** -23
    assert float(p.max()) > 0
