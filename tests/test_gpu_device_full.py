"""Calls with little device memory left: those that kept a smaller scratch, or none,
before they took the present forms fall back to forms with as little, with the
same bits."""
import numpy as np
import pytest

from conftest import geo, host

pytestmark = pytest.mark.gpu

ARGS = ("SO", "SD", "da", "na", "ai", "db", "nb", "bi", "nx", "ny", "nz")
MB = 1 << 20


class Full:
    """Holds device memory so that about `left` MB are free."""

    def __init__(self, torch, left):
        self.torch, self.left = torch, left

    def __enter__(self):
        torch = self.torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.held, step = [], 1 << 36
        while step >= 2 * MB:
            spare = torch.cuda.mem_get_info()[0] - self.left * MB
            n = min(step, spare) // (2 * MB) * (2 * MB)
            if n <= 0:
                break
            try:
                self.held.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                step //= 2
        free = torch.cuda.mem_get_info()[0]
        assert (self.left - 8) * MB <= free <= (self.left + 8) * MB, free

    def __exit__(self, *exc):
        del self.held
        self.torch.cuda.empty_cache()


@pytest.mark.parametrize("angle", [0.3, 1.5])
def test_projection_without_room_for_a_copy(torch_cuda, angle):
    import mcsart_b200 as m
    torch = torch_cuda
    g = geo(nx=320, ny=300, nz=301, na=70, nb=61, SO=900.0, SD=1350.0, da=6.5, db=7.2)
    a = [g[k] for k in ARGS]
    img = torch.rand((301, 300, 320), device="cuda")  # 115 MB
    want, got = (torch.full((61, 70), 7.0, device="cuda") for _ in range(2))
    with m.Context() as c:
        torch.cuda.synchronize()
        c.host_projection(want, img, angle, *a)
        c.synchronize()
    with m.Context() as c:
        small = geo()
        c.host_projection(torch.zeros((28, 40), device="cuda"), torch.zeros((16, 20, 24), device="cuda"),
                          angle, *[small[k] for k in ARGS])
        c.synchronize()
        with Full(torch, 64):
            c.host_projection(got, img, angle, *a)
            c.synchronize()
    np.testing.assert_array_equal(host(got), host(want))
    assert host(want).any()


def test_dvf_inverse_without_room_for_packed_displacements(torch_cuda):
    import mcsart_b200 as m
    torch = torch_cuda
    n = (224, 224, 200)  # 40 MB an array
    gen = torch.Generator(device="cuda").manual_seed(1)
    fields = torch.rand((6, n[2], n[1], n[0]), device="cuda", generator=gen) * 2 - 1
    want, got = (torch.zeros((3, n[2], n[1], n[0]), device="cuda") for _ in range(2))
    with m.Context() as c:
        torch.cuda.synchronize()
        c.invert_dvf(*want, *fields, 0.7, 0.3, *n, 5)
        c.synchronize()
    with m.Context() as c:
        c.invert_dvf(*got[:, :1, :1, :1].contiguous().cuda(), *fields, 0.7, 0.3, 1, 1, 1, 1)
        c.synchronize()
        with Full(torch, 136):  # between 3 and 4 arrays
            c.invert_dvf(*got, *fields, 0.7, 0.3, *n, 5)
            c.synchronize()
    np.testing.assert_array_equal(host(got), host(want))


def test_adjoint_without_room_for_the_rays_values(torch_cuda):
    import mcsart_b200 as m
    torch = torch_cuda
    # 64 MB of ray values and ratios, 32 MB of ratios; a few MB of tables
    g = geo(nx=40, ny=36, nz=33, na=2048, nb=2048, SO=120.0, SD=180.0, da=0.05, db=0.05)
    a = [g[k] for k in ARGS]
    proj = torch.rand((2048, 2048), device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))
    want, got = (torch.zeros((33, 36, 40), device="cuda") for _ in range(2))
    small = geo()
    with m.Context() as c:
        torch.cuda.synchronize()
        c.host_backprojection_adjoint(want, proj, 0.3, *a)
        c.synchronize()
    with m.Context() as c:
        c.host_backprojection_adjoint(torch.zeros((16, 20, 24), device="cuda"),
                                      torch.zeros((28, 40), device="cuda"), 0.3, *[small[k] for k in ARGS])
        c.synchronize()
        with Full(torch, 56):
            c.host_backprojection_adjoint(got, proj, 0.3, *a)
            c.synchronize()
    np.testing.assert_array_equal(host(got), host(want))
    assert host(want).any()
