"""get_interp_arrays_2D where the device has room for one component's scratch but
not for both at once: the same coefficients, one component after the other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_little_memory(nb):
    import torch
    nt, nx, ny = 100, 240, 200
    t, x, y = np.linspace(0, 1, nt), np.linspace(0, 1, nx), np.linspace(0, 1, ny)
    g = torch.Generator(device="cuda").manual_seed(1)
    U, V = (torch.rand((nt, nx, ny), generator=g, device="cuda", dtype=torch.float64) for _ in "uv")
    _, want_u, want_v = nb.get_interp_arrays_2D(t, x, y, U, V)
    want_u, want_v = want_u.cpu(), want_v.cpu()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    field = (nt + 2) * (nx + 2) * (ny + 2) * 8
    # the two inputs are there; both coefficient arrays and 2.5 fields more fit
    limit = torch.cuda.memory_reserved() + int(4.5 * field)
    torch.cuda.set_per_process_memory_fraction(limit / total)
    try:
        _, u, v = nb.get_interp_arrays_2D(t, x, y, U, V)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(u.cpu(), want_u) and torch.equal(v.cpu(), want_v)
