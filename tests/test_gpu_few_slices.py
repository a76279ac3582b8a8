"""Volumes of few slices: those of at most eight take the projector's copy a column
per thread."""
import numpy as np
import pytest

from conftest import dev, geo, host, rel_l2, volume
from test_gpu_aligned_copies import program, run  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu

ARGS = ("SO", "SD", "da", "na", "ai", "db", "nb", "bi", "nx", "ny", "nz")


@pytest.mark.parametrize("nz", [1, 2, 7, 8, 9])
def test_shallow_volumes_project_as_the_oracle(ctx, torch_cuda, oracle, nz):
    """1e-5 relative L2 (the bound of the parity tests); BF16 values are FP32
    values, so that their copy projects to the same bits."""
    import mcsart_b200 as m
    torch = torch_cuda
    g = geo(nx=37, ny=33, nz=nz, na=45, nb=2 * nz + 3, SO=120.0, SD=180.0, da=1.3, db=0.9)
    a = [g[k] for k in ARGS]
    v16 = dev(torch, volume((nz, 33, 37), seed=nz)).bfloat16()
    img = v16.float()
    for angle in (0.3, 1.5, 3.9):
        out = [torch.full((g["nb"], g["na"]), 7.0, device="cuda") for _ in range(3)]
        ctx.host_projection(out[0], img, angle, *a)
        ctx.projection_ex(out[1], v16, angle, *a, fp_sum=0)
        m.projection_noalloc(out[2], img, angle, *a, stream=torch.cuda.current_stream())
        ctx.synchronize()
        torch.cuda.synchronize()
        o = oracle.projection(host(img), angle, g)
        assert np.linalg.norm(o) > 0 and rel_l2(host(out[0]), o) <= 1e-5
        np.testing.assert_array_equal(host(out[1]), host(out[0]))
        np.testing.assert_array_equal(host(out[2]), host(out[0]))


def test_one_slice_has_the_plain_loops_bits(program):
    """A slice's edges lie at 0 and 1 of the axial coordinate, where footprints may
    begin or end exactly, or within a rounding of it."""
    cases = []
    for nb, bi in ((1, 0.0), (2, 0.0), (5, 0.0), (40, 0.0), (3, 0.4), (2, 0.5), (4, -1e-7)):
        g = geo(nx=41, ny=37, nz=1, na=33, nb=nb, SO=90.0, SD=135.0, da=1.1, db=0.7, bi=bi)
        cases += [(g, nzp, angle) for nzp in (1, 2)
                  for angle in (0.0, 0.3, 0.7853982, 1.5, 1.5707964, 3.9)]
    run(program, cases)
