"""ftle_from_eig of views that are no plain memory: a lazily negated one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_lazily_negated_view(nb):
    import torch
    a = torch.linspace(-30.0, 30.0, 35 * 21, dtype=torch.float64, device="cuda").reshape(35, 21)
    e = torch.complex(torch.zeros_like(a), a).conj().imag
    assert e.is_neg()
    want = np.where(-a.cpu().numpy() > 1.0, np.log(np.maximum(-a.cpu().numpy(), 1.0)) / 6.0, 0.0)
    np.testing.assert_allclose(nb.ftle_from_eig(e, -3.0).cpu().numpy(), want, rtol=1e-14, atol=0)
    np.testing.assert_allclose(nb.ftle_from_eig(e[3:9, 2], -3.0).cpu().numpy(), want[3:9, 2],
                               rtol=1e-14, atol=0)
