"""Launchers whose scratch belongs to the context, called on two streams in turn
without a synchronize: each call's results are those of the same call alone."""
import numpy as np
import pytest

from conftest import dev, geo, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("angle", [0.3, 1.5])
def test_calls_in_turn_on_two_streams_do_not_share_scratch(torch_cuda, angle):
    import mcsart_b200 as m
    torch = torch_cuda
    g = geo(nx=144, ny=128, nz=120, na=180, nb=150, SO=300.0, SD=450.0, da=1.3, db=1.2)
    a = [g[k] for k in ("SO", "SD", "da", "na", "ai", "db", "nb", "bi", "nx", "ny", "nz")]
    assert 144 * 128 * 120 >= 1 << 21  # the backprojector that keeps scratch
    rng = np.random.default_rng(8)
    imgs = [dev(torch, rng.random((120, 128, 144), dtype=np.float32)) for _ in range(4)]
    projs = [dev(torch, rng.random((150, 180), dtype=np.float32)) for _ in range(4)]
    calls = [("host_projection", imgs, (150, 180)), ("host_backprojection", projs, (120, 128, 144)),
             ("host_backprojection_adjoint", projs, (120, 128, 144))]
    ctx = m.Context()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for name, ins, shape in calls:
        call = getattr(ctx, name)
        alone, turn = ([torch.zeros(shape, device="cuda") for _ in range(12)] for _ in range(2))
        torch.cuda.synchronize()
        for i in range(12):
            call(alone[i], ins[i % 4], angle, *a)
            ctx.synchronize()
        for i in range(12):
            ctx.set_stream(streams[i % 2])
            call(turn[i], ins[i % 4], angle, *a)
        torch.cuda.synchronize()
        for x, y in zip(alone, turn):
            np.testing.assert_array_equal(host(x), host(y))


@pytest.mark.parametrize("angle", [0.3, 1.5])  # x-driven and y-driven rays
def test_projections_captured_on_a_new_context(torch_cuda, angle):
    """The graph owns the volume's copy: a first call can be captured, and later
    calls with larger volumes leave the graph's results alone."""
    import mcsart_b200 as m
    torch = torch_cuda
    g, big = (geo(nx=n, ny=n, nz=n, na=48, nb=40, SO=120.0, SD=180.0, da=1.2, db=1.2)
              for n in (33, 64))
    a, b = ([q[k] for k in ("SO", "SD", "da", "na", "ai", "db", "nb", "bi", "nx", "ny", "nz")]
            for q in (g, big))
    rng = np.random.default_rng(9)
    img = dev(torch, rng.random((33, 33, 33), dtype=np.float32))
    large = dev(torch, rng.random((64, 64, 64), dtype=np.float32))
    eager, sums, got, got_sums, other = (torch.zeros((40, 48), device="cuda") for _ in range(5))
    warm, s = m.Context(), torch.cuda.Stream()
    warm.host_projection(eager, img, angle, *a)  # (also loads the kernels' code)
    warm.projection_ex(sums, img, angle, *a, fp_sum=2)
    warm.synchronize()
    ctx = m.Context(stream=s)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ctx.host_projection(got, img, angle, *a)
        ctx.projection_ex(got_sums, img, angle, *a, fp_sum=2)
    for _ in range(2):
        ctx.host_projection(other, large, angle, *b)
        ctx.synchronize()
        got.zero_(), got_sums.zero_()
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(host(got), host(eager))
        np.testing.assert_array_equal(host(got_sums), host(sums))
