"""The slice-lane backprojector against bp_kernel and the FP64 oracle.

mcsart_backprojection takes it from 2^21 voxels on; every voxel's sum has the
same operations in the same order in both kernels, so the middle slices of a
volume above the line equal the volume below it that they make.
"""
import numpy as np
import pytest

from conftest import dev, geo, host, rel_l2

pytestmark = pytest.mark.gpu

MIN = 1 << 21  # BP_SLICE_LANES_MIN


def _args(g):
    return (g["SO"], g["SD"], g["da"], g["na"], g["ai"], g["db"], g["nb"], g["bi"], g["nx"],
            g["ny"], g["nz"])


def _bp(ctx, torch, proj, a, g):
    out = torch.full((g["nz"], g["ny"], g["nx"]), 7.0, device="cuda")
    ctx.host_backprojection(out, dev(torch, proj), a, *_args(g))
    ctx.synchronize()
    return host(out)


# depths with full, half-empty and nearly empty last tiles; odd rows; wide
# voxels (more than four rows each); a source too close for the proof
@pytest.mark.parametrize("nx,ny,nz,na,nb,kw", [
    (181, 173, 67, 97, 51, {}), (160, 160, 96, 64, 64, {}), (129, 131, 129, 75, 80, dict(db=0.3)),
    (200, 180, 82, 90, 61, dict(SO=138.0, SD=207.0, da=3.0, db=2.0))])
def test_larger_volume_equals_its_slabs_of_slices(ctx, torch_cuda, nx, ny, nz, na, nb, kw):
    torch = torch_cuda
    assert nx * ny * nz >= MIN
    g = geo(nx=nx, ny=ny, nz=nz, na=na, nb=nb, **{**dict(SO=300.0, SD=450.0, da=2.9, db=2.3), **kw})
    rng = np.random.default_rng(nx)
    proj = rng.random((nb, na), dtype=np.float32)
    proj[0, :3] = 1e-40  # denormal texels read as zeros
    for a in (0.3, 0.7853982, 2.4):
        big = _bp(ctx, torch, proj, a, g)
        # its middle 40 slices are a volume of their own with the same centre plane
        assert nx * ny * 40 < MIN
        small = _bp(ctx, torch, proj, a, dict(g, nz=40))
        np.testing.assert_array_equal(big[nz // 2 - 20: nz // 2 + 20], small)


def test_larger_volume_matches_the_oracle(ctx, torch_cuda, oracle):
    torch = torch_cuda
    g = geo(nx=130, ny=128, nz=127, na=80, nb=70, SO=300.0, SD=450.0, da=2.9, db=2.9)
    proj = np.random.default_rng(3).random((70, 80), dtype=np.float32)
    for a in (0.3, 2.4):
        assert rel_l2(_bp(ctx, torch, proj, a, g), oracle.backprojection(proj, a, g)) <= 1e-4


def test_capture_on_a_new_context_needs_no_scratch(torch_cuda):
    """A captured call takes bp_kernel, which keeps no workspace: the same bits."""
    import mcsart_b200 as m
    torch = torch_cuda
    g = geo(nx=128, ny=128, nz=128, na=80, nb=70, SO=300.0, SD=450.0, da=2.9, db=2.9)
    proj = dev(torch, np.random.default_rng(4).random((70, 80), dtype=np.float32))
    eager, captured = (torch.full((128, 128, 128), 7.0, device="cuda") for _ in range(2))
    s = torch.cuda.Stream()
    ctx = m.Context(stream=s)
    # (a smaller volume first, so that the kernel's code is loaded)
    small = torch.empty((8, 128, 128), device="cuda")
    torch.cuda.synchronize()
    ctx.host_backprojection(small, proj, 0.3, *_args(dict(g, nz=8)))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ctx.host_backprojection(captured, proj, 0.3, *_args(g))
    ctx.host_backprojection(eager, proj, 0.3, *_args(g))
    ctx.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(host(captured), host(eager))
