"""A data point of infinite variance takes no part in the log-likelihood without its
log-determinant, nor in its gradients: against the solve without that row, at
sizes of several CTAs, the point first, between others and last.

Tolerance as for the finite blocks (condition number about 30): 1e-12.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

import jax_cosmo_gb300 as jc  # noqa: E402

TOL = 1e-12


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def blocks(n, nd, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, _ = torch.linalg.qr(torch.randn(nd, n, n, dtype=torch.float64, device="cuda", generator=g))
    a = (q * torch.linspace(1.0, 30.0, n, dtype=torch.float64, device="cuda")) @ q.transpose(-1, -2)
    return 0.5 * (a + a.transpose(-1, -2)), torch.randn(n * nd, dtype=torch.float64, device="cuda", generator=g)


@pytest.mark.parametrize("n,at", [(1, 0), (6, 0), (6, 3), (6, 5), (30, 17), (55, 0), (60, 59)])
@pytest.mark.parametrize("dense", [False, True])
def test_masked_point(n, at, dense):
    nd, l = 3, 1
    a, mu = blocks(n, nd, n + at)
    a[l, at, at] = float("inf")
    r = mu.reshape(n, nd).T  # data 0
    want, dmu = 0.0, torch.zeros(nd, n, dtype=torch.float64, device="cuda")
    for q in range(nd):
        keep = [i for i in range(n) if not (q == l and i == at)]
        if keep:
            x = torch.linalg.solve(a[q][keep][:, keep], r[q][keep])
            want = want - 0.5 * float(r[q][keep] @ x)
            dmu[q, keep] = -x
    C = a.permute(1, 2, 0).contiguous()
    if dense:
        d = torch.zeros(n, nd, n, nd, dtype=torch.float64, device="cuda")
        i = torch.arange(nd, device="cuda")
        d[:, i, :, i] = a
        C = d.reshape(n * nd, n * nd)
        C._jcg_n_ell = nd
    m, data = mu.clone().requires_grad_(True), torch.zeros_like(mu)
    v = jc.likelihood.gaussian_log_likelihood(data, m, C, include_logdet=False)
    assert abs(float(v.detach()) - want) <= TOL * max(abs(want), 1.0)
    assert float(jc.likelihood.gaussian_log_likelihood(data, mu, C, include_logdet=False)) == float(v.detach())
    (g,) = torch.autograd.grad(v, m)
    g = g.reshape(n, nd).T
    assert float(g[l, at]) == 0.0 and float((g - dmu).abs().max()) <= TOL * max(float(dmu.abs().max()), 1.0)
    assert float(jc.likelihood.gaussian_log_likelihood(data, mu, C, include_logdet=True)) == float("inf")


def test_gradient_in_the_covariance():
    a, mu = blocks(5, 3, 2)
    a[1, 2, 2] = float("inf")
    C = a.permute(1, 2, 0).contiguous().requires_grad_(True)
    v = jc.likelihood.gaussian_log_likelihood(torch.zeros_like(mu), mu, C, include_logdet=False)
    (g,) = torch.autograd.grad(v, C)
    assert bool(torch.isfinite(g).all())
    assert float(g[2, :, 1].abs().max()) == 0.0 and float(g[:, 2, 1].abs().max()) == 0.0


@pytest.mark.parametrize("bad", [0.0, -1.0, float("-inf"), float("nan")])
def test_other_pivots_stay_refused(bad):
    a, mu = blocks(4, 3, 9)
    a[2] = torch.eye(4, dtype=torch.float64, device="cuda")
    a[2, 1, 1] = bad
    v = jc.likelihood.gaussian_log_likelihood(torch.zeros_like(mu), mu, a.permute(1, 2, 0).contiguous(), include_logdet=False)
    assert bool(torch.isnan(v))
