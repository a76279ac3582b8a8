"""Odd depths: columns of the z-fastest copies are a slice longer than the volume,
and whatever writes them writes zero there.  Results must not depend on what the
buffers held, and the copy without the added slice (a volume that fills
mcsart_projection_noalloc's scratch) must project to the same bits."""
import numpy as np
import pytest

from conftest import dev, geo, host, rel_l2, volume
from test_gpu_sart import make_case

pytestmark = pytest.mark.gpu

ARGS = ("SO", "SD", "da", "na", "ai", "db", "nb", "bi", "nx", "ny", "nz")


def _run(m, torch, ctx, case, **opt):
    g, it, img0, proj, F = case
    dt = {0: torch.float32, 1: torch.bfloat16, 2: torch.float16}[opt["storage"]]
    img, resid = dev(torch, img0), torch.zeros((it["n_views"], g["nb"], g["na"]), device="cuda")
    fields = dev(torch, np.stack(F)).to(dt)
    op = np.array([1, 0, 1], np.int32)
    ctx.aumisart_device(geo=g, n_views=it["n_views"], lambda_=1.0, angles=it["angles"],
                        volumes=it["volumes"], flows=it["flows"], img=img,
                        proj=dev(torch, proj).to(dt), norm=torch.zeros(3 * it["n_views"], device="cuda"),
                        resid=resid, fields=fields, n_iter=3, op_iter=op,
                        options=m.default_options(**opt))
    ctx.synchronize()
    return [host(img), host(resid), host(fields.float())]


@pytest.mark.parametrize("opt", [dict(storage=0), dict(storage=2), dict(storage=1, subset=2),
                                 dict(storage=0, fp_sum=2)])
@pytest.mark.parametrize("nz", [15, 17])
def test_odd_depth_ignores_what_the_buffers_held(torch_cuda, oracle, nz, opt):
    import mcsart_b200 as m
    torch = torch_cuda
    op = (1, 0, 1)
    odd = make_case(oracle, motion=True, nx=20, ny=20, nz=nz, op_iter=op, seed=4)
    g, it, img0, proj, F = make_case(oracle, motion=True, nx=24, ny=24, nz=20, op_iter=op, seed=5)
    fresh, used = m.Context(), m.Context()
    _run(m, torch, used, (g, it, np.full_like(img0, np.nan), proj, F), **opt)
    for a, b in zip(_run(m, torch, fresh, odd, **opt), _run(m, torch, used, odd, **opt)):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)


def test_copy_without_the_added_slice_projects_to_the_same_bits(ctx, torch_cuda):
    import mcsart_b200 as m
    torch = torch_cuda
    g = geo(nx=568, ny=567, nz=13, na=70, nb=33, SO=1700.0, SD=2550.0, da=12.0, db=0.9)
    a = [g[k] for k in ARGS]
    n = g["nx"] * g["ny"]
    assert n * 13 <= 4194304 < n * 14  # MCSART_NOALLOC_MAX_VOXELS
    img = dev(torch, volume((13, 567, 568), seed=6))
    for angle in (0.3, 1.5):
        outs = [torch.full((g["nb"], g["na"]), 7.0, device="cuda") for _ in range(2)]
        ctx.host_projection(outs[0], img, angle, *a)
        m.projection_noalloc(outs[1], img, angle, *a, stream=torch.cuda.current_stream())
        ctx.synchronize()
        torch.cuda.synchronize()
        assert host(outs[0]).any()
        np.testing.assert_array_equal(host(outs[0]), host(outs[1]))


@pytest.mark.parametrize("nz", [63, 65, 128, 129])
def test_depths_around_the_copy_s_tile_match_the_oracle(ctx, torch_cuda, oracle, nz):
    """The copy turns 32 columns by 64 slices at a time (1e-5 relative L2: the
    bound of the parity tests)."""
    torch = torch_cuda
    g = geo(nx=33, ny=5, nz=nz, na=20, nb=150, SO=120.0, SD=180.0, da=3.0, db=1.7)
    img = volume((nz, 5, 33), seed=nz)
    out = torch.full((g["nb"], g["na"]), 7.0, device="cuda")
    for a in (0.3, 1.5):
        ctx.host_projection(out, dev(torch, img), a, *[g[k] for k in ARGS])
        ctx.synchronize()
        o = oracle.projection(img, a, g)
        assert np.linalg.norm(o) > 0 and rel_l2(host(out), o) <= 1e-5, (a, rel_l2(host(out), o))
