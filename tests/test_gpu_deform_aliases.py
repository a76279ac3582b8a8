"""kernel_forwardDVF's outputs in place of its fields: each component is computed and
stored before the next one's fields are read."""
import numpy as np
import pytest

from conftest import dev, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [8, 7])
@pytest.mark.parametrize("places", [(0, 1, 2), (1, 2, 0), (4, 1, 2), (2, 5, 0), (3, 4, 5), (1, 4, 5)])
def test_forward_dvf_over_its_own_fields(ctx, torch_cuda, nx, places):
    """places[c]: the field (alpha_x .. beta_z) that component c is written over; the
    sums are exact (small integers)."""
    torch = torch_cuda
    f = np.random.default_rng(sum(places)).integers(-50, 50, (6, 4, 5, nx)).astype(np.float32)
    want = f.copy()
    for c in range(3):
        want[places[c]] = want[c] * 2 + want[3 + c] * 3
    d = [dev(torch, x) for x in f]
    ctx.kernel_forwardDVF(*[d[p] for p in places], *d, 2.0, 3.0, nx, 5, 4)
    ctx.synchronize()
    for got, w in zip(d, want):
        np.testing.assert_array_equal(host(got), w)
