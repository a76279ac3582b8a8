"""A stream that is destroyed with work under way, and the next one, which may get
its handle: the context's scratch stays ordered across them."""
import ctypes

import numpy as np
import pytest

from conftest import geo, host

pytestmark = pytest.mark.gpu


def test_calls_on_streams_created_and_destroyed_in_turn(torch_cuda):
    import mcsart_b200 as m
    torch = torch_cuda
    # the library's own runtime calls are linked in; these are the installed runtime's
    rt = ctypes.CDLL("libcudart.so.12")
    g = geo(nx=144, ny=128, nz=120, na=180, nb=150, SO=300.0, SD=450.0, da=1.3, db=1.2)
    a = [g[k] for k in ("SO", "SD", "da", "na", "ai", "db", "nb", "bi", "nx", "ny", "nz")]
    gen = torch.Generator(device="cuda").manual_seed(8)
    imgs = [torch.rand((120, 128, 144), device="cuda", generator=gen) for _ in range(4)]
    alone, turn = ([torch.zeros((150, 180), device="cuda") for _ in range(24)] for _ in range(2))
    ctx = m.Context()
    torch.cuda.synchronize()
    for i, o in enumerate(alone):
        ctx.host_projection(o, imgs[i % 4], 0.3, *a)
        ctx.synchronize()
    for i, o in enumerate(turn):
        s = ctypes.c_void_p()
        assert rt.cudaStreamCreateWithFlags(ctypes.byref(s), 1) == 0
        ctx.set_stream(s.value)
        ctx.host_projection(o, imgs[i % 4], 0.3, *a)
        assert rt.cudaStreamDestroy(s) == 0  # returns with the call under way
    ctx.set_stream(0)
    torch.cuda.synchronize()
    for x, y in zip(alone, turn):
        np.testing.assert_array_equal(host(x), host(y))
