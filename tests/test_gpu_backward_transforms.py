"""The log-likelihood's gradient in a batch of sparse covariances under a vectorised
Jacobian and with a forward tangent in the cotangent, by the library.
Tolerance: the two forms round a product and an inverse apart: 1e-12 of the largest entry."""
import pytest
import torch
from torch.autograd import forward_ad as fw

pytestmark = pytest.mark.gpu

import jax_cosmo_gb300 as jc  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def inputs():
    g = torch.Generator().manual_seed(1)
    a = torch.randn(3, 7, 5, 5, dtype=torch.float64, generator=g)
    C = (a @ a.transpose(-1, -2) + 5 * torch.eye(5, dtype=torch.float64)).permute(0, 2, 3, 1).contiguous()
    return [torch.randn(3, 35, dtype=torch.float64, generator=g).cuda() for _ in range(2)] + [C.cuda()]


@pytest.mark.parametrize("logdet", [True, False])
def test_jacobian_in_the_covariance(logdet):
    data, mu, C = inputs()
    f = lambda c: jc.likelihood.gaussian_log_likelihood(data, mu, c, include_logdet=logdet)  # noqa: E731
    one = torch.autograd.functional.jacobian(f, C)
    got = torch.autograd.functional.jacobian(f, C, vectorize=True)
    assert float((got - one).abs().max()) < 1e-12 * float(one.abs().max())


def test_forward_tangent_of_the_cotangent():
    data, mu, C = inputs()
    x = C.requires_grad_(True)
    ll = jc.likelihood.gaussian_log_likelihood(data, mu, x)
    go, dgo = torch.tensor([[0.3, -1.0, 2.0], [1.0, 0.5, -0.2]], dtype=torch.float64).cuda()
    (want,) = torch.autograd.grad(ll, x, dgo, retain_graph=True)
    with fw.dual_level():
        (g,) = torch.autograd.grad(ll, x, fw.make_dual(go, dgo))
        t = fw.unpack_dual(g).tangent
        assert t is not None and float((t - want).abs().max()) < 1e-12 * float(want.abs().max())
