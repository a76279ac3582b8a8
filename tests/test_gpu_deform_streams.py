"""Warps through the texture, whose 3D array the context keeps, and the loop, whose
working volumes it keeps, on two streams in turn without a synchronize: each
call's results are those of the same call alone.  The volumes are large enough
for a call to be under way when the next is made."""
import numpy as np
import pytest

from conftest import dev, host
from test_gpu_sart import make_case

pytestmark = pytest.mark.gpu


def _in_turn(torch, ctx, call, outs):
    """call(i, out) for every i, alone and in turn on two streams."""
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    alone, turn = outs(), outs()
    torch.cuda.synchronize()
    for i, o in enumerate(alone):
        call(i, o)
        ctx.synchronize()
    for i, o in enumerate(turn):
        ctx.set_stream(streams[i % 2])
        call(i, o)
    torch.cuda.synchronize()
    for a, t in zip(alone, turn):
        np.testing.assert_array_equal(host(a), host(t))


@pytest.mark.parametrize("ex", [False, True])
def test_texture_warps_in_turn_on_two_streams(torch_cuda, ex):
    import mcsart_b200 as m
    torch = torch_cuda
    n = 288
    gen = torch.Generator(device="cuda").manual_seed(3)
    imgs = [torch.rand((n, n, n), device="cuda", generator=gen) for _ in range(3)]
    fields = torch.rand((6, n, n, n), device="cuda", generator=gen) * 4 - 2
    ctx = m.Context()

    def call(i, out):
        if ex:
            ctx.deform_ex(out, imgs[i % 3], n, n, n, 0.7, 0.3, fields, interp=m.INTERP_TEXTURE)
        else:
            ctx.host_deform(out, imgs[i % 3], n, n, n, 0.7, 0.3, *fields)

    _in_turn(torch, ctx, call, lambda: [torch.zeros((n, n, n), device="cuda") for _ in range(8)])


def test_loops_in_turn_on_two_streams(torch_cuda, oracle):
    import mcsart_b200 as m
    torch = torch_cuda
    cases = [make_case(oracle, motion=True, nx=48, ny=48, nz=40, na=64, nb=56, op_iter=(1,), seed=s)
             for s in (2, 3)]
    ins = [(g, it, dev(torch, i), dev(torch, p), dev(torch, np.stack(F))) for g, it, i, p, F in cases]
    ctx = m.Context()

    def call(i, img):
        g, it, img0, proj, fields = ins[i % 2]
        ctx.aumisart_device(geo=g, n_views=it["n_views"], lambda_=1.0, angles=it["angles"],
                            volumes=it["volumes"], flows=it["flows"], img=img, proj=proj,
                            fields=fields, n_iter=1, op_iter=np.array([1], np.int32),
                            options=m.default_options(use_graph=0))

    _in_turn(torch, ctx, call, lambda: [ins[i % 2][2].clone() for i in range(6)])
