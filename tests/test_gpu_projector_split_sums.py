"""The split-sum projector (plain and Kahan sums, FP32 and FP64 geometry) at the
edges of its slab tables.

A warp of fp_kernel is 32 detector rows of one column and a table 32 slabs of
its slab group; footprints of more than two voxels or slices take weights of
their own.  Each shape is checked against the FP64 oracle with the bound of the
parity tests (1e-5 relative L2: up to 256 slabs of terms rounded to 2^-24 each).
"""
import numpy as np
import pytest

from conftest import dev, geo, host, rel_l2, volume

pytestmark = pytest.mark.gpu

# (nx, ny, nz, na, nb, da, db): one slab, 31 to 33 and 65 slabs, one group and
# several (na * ceil(nb / 32) small), rows past the last warp, wide footprints
SHAPES = [(1, 1, 1, 2, 2, 0.9, 0.8), (33, 31, 2, 3, 31, 0.9, 0.8), (32, 32, 1, 4, 32, 0.9, 0.8),
          (31, 65, 3, 5, 33, 0.9, 0.8), (40, 36, 40, 170, 290, 0.3, 0.2),
          (40, 36, 40, 17, 40, 1.1, 1.6), (24, 40, 21, 33, 40, 2.7, 3.9)]


@pytest.mark.parametrize("geom64", [0, 1])
@pytest.mark.parametrize("fp_sum", [1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_split_sums_match_the_oracle(ctx, torch_cuda, oracle, shape, fp_sum, geom64):
    torch = torch_cuda
    nx, ny, nz, na, nb, da, db = shape
    g = geo(nx=nx, ny=ny, nz=nz, na=na, nb=nb, SO=90.0, SD=135.0, da=da, db=db, ai=0.37, bi=-0.61)
    img = volume((nz, ny, nx), seed=nx)
    d_img, out = dev(torch, img), torch.full((nb, na), 7.0, device="cuda")
    for a in (0.3, 1.5, 3.9, 5.2):
        ctx.projection_ex(out, d_img, a, g["SO"], g["SD"], g["da"], g["na"], g["ai"], g["db"],
                          g["nb"], g["bi"], nx, ny, nz, fp_sum=fp_sum, geom64=geom64)
        ctx.synchronize()
        o = oracle.projection(img, a, g)
        assert np.linalg.norm(o) > 0 and rel_l2(host(out), o) <= 1e-5, (a, rel_l2(host(out), o))
