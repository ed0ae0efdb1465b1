"""ftle_from_eig reads eigenvalues of any layout: the strided views that it
takes in place give what their C-ordered copies give."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("view", [
    lambda t: t[..., 1], lambda t: t[..., 0], lambda t: t[1:, :, 1], lambda t: t[:, 1:-1, 1],
    lambda t: t[::2, :, 1], lambda t: t[..., 1].T, lambda t: t[:, 3, 1], lambda t: t[4, :, 1],
    lambda t: t[4, :, 1:], lambda t: t[4:5, :, 1], lambda t: t[:, 3:4, 1], lambda t: t[2, 3, 1],
    lambda t: t[2, 3, 1].expand(6), lambda t: t[:0, :, 1], lambda t: t,
    lambda t: t[..., 1].float(), lambda t: t[..., 1].cpu()])
def test_views(nb, view):
    import torch
    rng = np.random.default_rng(5)
    t = torch.from_numpy(np.exp(rng.uniform(-3, 9, (37, 29, 2)))).cuda()
    v = view(t)
    got = nb.ftle_from_eig(v, -7.0)
    want = nb.ftle_from_eig(v.to(torch.float64).cpu().numpy().copy(), -7.0)
    assert tuple(got.shape) == tuple(v.shape) and got.is_contiguous()
    np.testing.assert_array_equal(got.cpu().numpy(), want)
