"""Detectors of few rows: the split-sum projector's warps are then 32 columns of a
row instead of 32 rows of a column.  A ray's sum does not depend on it, so that
one row by itself has the bits of the same row of a tall detector."""
import numpy as np
import pytest

from conftest import dev, geo, host, rel_l2, volume

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geom64", [0, 1])
@pytest.mark.parametrize("fp_sum", [1, 2])
# (nx, ny, nz, na, da): driving axes in one warp at 0.7853982, columns past the last warp
@pytest.mark.parametrize("shape", [(64, 64, 20, 70, 0.9), (72, 65, 1, 33, 1.9), (65, 80, 9, 31, 0.4)])
def test_one_row_has_the_bits_of_a_tall_detector_s(ctx, torch_cuda, oracle, shape, fp_sum, geom64):
    torch = torch_cuda
    nx, ny, nz, na, da = shape
    img = volume((nz, ny, nx), seed=nx)
    d_img = dev(torch, img)

    def project(g, a):
        out = torch.full((g["nb"], g["na"]), 7.0, device="cuda")
        ctx.projection_ex(out, d_img, a, g["SO"], g["SD"], g["da"], g["na"], g["ai"], g["db"],
                          g["nb"], g["bi"], nx, ny, nz, fp_sum=fp_sum, geom64=geom64)
        ctx.synchronize()
        return host(out)

    tall = geo(nx=nx, ny=ny, nz=nz, na=na, nb=64, SO=190.0, SD=285.0, da=da, db=0.5)
    for a in (0.3, 0.7853982, 1.5, 3.9):
        t = project(tall, a)
        assert rel_l2(t, oracle.projection(img, a, tall)) <= 1e-5
        for rows in ((31,), (30, 31, 32)):
            one = dict(tall, nb=len(rows), bi=tall["bi"] + rows[0])
            np.testing.assert_array_equal(project(one, a), t[list(rows)])
