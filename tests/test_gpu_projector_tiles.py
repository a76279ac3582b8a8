"""The row-lane projector at the edges of its tiles and of its fast form.

A warp of fp_ref_kernel is 32 detector rows of one column, a block four
columns, a table 32 slabs, a stage two to eight; windows begin on even slices
where the depth is even and are copied slice by slice where it is odd.  Rays
whose footprint spans more than two slices, or whose 32 rows span more than a
window, take the direct or the general form.  Each shape is checked against the
FP64 oracle with the bound of the parity tests (1e-5 relative L2: 256 slabs of
terms rounded to 2^-24 each), and forms that must agree are compared bit for bit.
"""
import numpy as np
import pytest

from conftest import dev, geo, host, rel_l2, volume

pytestmark = pytest.mark.gpu

ANGLES = [0.3, 0.7853982, 1.5, 3.9, 5.2]


def _args(g):
    return (g["SO"], g["SD"], g["da"], g["na"], g["ai"], g["db"], g["nb"], g["bi"], g["nx"],
            g["ny"], g["nz"])


# (nx, ny, nz, na, nb, da, db): remainders of rows, columns, slabs and depth;
# db = 1.6: more than two slices at a slab; db = 1.45: 32 rows wider than a window
SHAPES = [(33, 31, 2, 3, 31, 0.9, 0.8), (32, 32, 1, 4, 32, 0.9, 0.8), (31, 65, 3, 5, 33, 0.9, 0.8),
          (64, 24, 17, 9, 65, 0.7, 0.7), (40, 40, 48, 21, 64, 0.9, 1.45),
          (40, 36, 40, 17, 40, 1.1, 1.6), (24, 40, 21, 33, 40, 2.7, 1.3), (5, 7, 64, 6, 97, 0.3, 0.9)]


@pytest.mark.parametrize("shape", SHAPES)
def test_projection_at_tile_edges_matches_the_oracle(ctx, torch_cuda, oracle, shape):
    torch = torch_cuda
    nx, ny, nz, na, nb, da, db = shape
    g = geo(nx=nx, ny=ny, nz=nz, na=na, nb=nb, SO=90.0, SD=135.0, da=da, db=db, ai=0.37, bi=-0.61)
    img = volume((nz, ny, nx), seed=nx)
    d_img = dev(torch, img)
    views = torch.zeros((len(ANGLES), nb, na), device="cuda")
    ctx.projection_views(views, d_img, ANGLES, *_args(g))
    for a, v in zip(ANGLES, views):
        out = torch.full((nb, na), 7.0, device="cuda")
        ctx.host_projection(out, d_img, a, *_args(g))
        ctx.synchronize()
        o = oracle.projection(img, a, g)
        assert np.linalg.norm(o) > 0 and rel_l2(host(out), o) <= 1e-5, (a, rel_l2(host(out), o))
        np.testing.assert_array_equal(host(v), host(out))


@pytest.mark.parametrize("nz", [16, 17])
@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
def test_16bit_volume_projects_as_the_same_values_in_fp32(ctx, torch_cuda, nz, dtype):
    """Every 16-bit value is an FP32 value, and the sums are FP32 either way."""
    torch = torch_cuda
    g = geo(nx=40, ny=36, nz=nz, na=37, nb=45, SO=90.0, SD=135.0)
    v16 = dev(torch, volume((nz, 36, 40), seed=5)).to(getattr(torch, dtype))
    for a in ANGLES:
        p16, p32 = (torch.zeros((g["nb"], g["na"]), device="cuda") for _ in range(2))
        ctx.projection_ex(p16, v16, a, *_args(g), fp_sum=0)
        ctx.host_projection(p32, v16.float(), a, *_args(g))
        ctx.synchronize()
        np.testing.assert_array_equal(host(p16), host(p32))


@pytest.mark.parametrize("nz", [64, 63])
def test_voxels_no_ray_meets_leave_no_trace(ctx, torch_cuda, nz):
    """Slices the detector does not cover, and those beside the ones it covers,
    hold infinities and NaN; the projections are those with zeros there."""
    torch = torch_cuda
    g = geo(nx=32, ny=32, nz=nz, na=48, nb=8, SO=90.0, SD=135.0, da=0.9, db=0.8)
    img = volume((nz, 32, 32), seed=8)
    # rows reach z2 = 4 * 0.8 on the detector: at most 3.2 * (90 + 23) / 135 < 3
    # voxels from the centre plane on any slab
    outside = np.abs(np.arange(nz) + 0.5 - nz // 2) > 4.0
    p = []
    for fill in (0.0, np.inf, np.nan):
        img[outside] = fill
        for a in ANGLES:
            out = torch.zeros((g["nb"], g["na"]), device="cuda")
            ctx.host_projection(out, dev(torch, img), a, *_args(g))
            ctx.synchronize()
            p.append(host(out))
    assert all(np.isfinite(x).all() and (x != 0).any() for x in p)
    for k, x in enumerate(p[len(ANGLES):]):
        np.testing.assert_array_equal(x, p[k % len(ANGLES)])
