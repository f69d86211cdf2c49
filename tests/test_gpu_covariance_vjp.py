"""Backward of the Gaussian covariance by its kernel against torch autograd of the
formula, over tracer counts (1 to 16), ell counts around the CTA's 128 threads, both
forms, batches, and each kind of noise; the gradient under create_graph, which
stays in torch operations; and the log-likelihood's gradient in a batch of sparse
covariances.

Tolerance: a sum of at most 512 products of random sign: 1e-13 of the largest entry.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import jax_cosmo_gb300 as jc  # noqa: E402
from jax_cosmo_gb300 import autodiff  # noqa: E402
from jax_cosmo_gb300.angular_cl import _get_cov_blocks_ordering  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


class _P:
    def __init__(self, n):
        self.n_tracers = n


def plain(ell, n_tr, cl, noise, f_sky):
    """[B, n_cls, n_cls, n_ell] of angular_cl.py:134-162"""
    b = torch.tensor(_get_cov_blocks_ordering([_P(n_tr)]), device=cl.device)
    o = cl + noise
    norm = torch.as_tensor((2 * ell + 1) * np.gradient(ell) * f_sky, device=cl.device)
    c = (o[:, b[:, 0]] * o[:, b[:, 1]] + o[:, b[:, 2]] * o[:, b[:, 3]]) / norm
    n = cl.shape[1]
    return c.reshape(cl.shape[0], n, n, -1)


@pytest.mark.parametrize("n_tr,n_ell,B", [(1, 2, 1), (2, 128, 3), (5, 129, 2), (16, 3, 1)])
@pytest.mark.parametrize("sparse", [True, False])
@pytest.mark.parametrize("noise", ["none", "cl", "tracer"])
def test_backward(n_tr, n_ell, B, sparse, noise):
    gen = torch.Generator().manual_seed(n_tr)
    n = n_tr * (n_tr + 1) // 2
    ell = np.geomspace(10, 3000, n_ell)
    cl = torch.rand(B, n, n_ell, generator=gen, dtype=torch.float64).cuda()
    cn = torch.rand(n, n_ell, generator=gen, dtype=torch.float64) if noise == "cl" else None
    tn = torch.rand(n_tr, generator=gen, dtype=torch.float64) if noise == "tracer" else None
    nz = torch.zeros(n, n_ell, dtype=torch.float64)
    if cn is not None:
        nz = cn
    if tn is not None:
        k = 0
        for i in range(n_tr):
            nz[k] = tn[i]
            k += n_tr - i
    ref_in = cl.clone().requires_grad_(True)
    w = torch.randn(B, n, n, n_ell, generator=gen, dtype=torch.float64).cuda()
    ref, = torch.autograd.grad((plain(ell, n_tr, ref_in, nz.cuda(), 0.3) * w).sum(), ref_in)
    x = cl.clone().requires_grad_(True)
    cov = autodiff.covariance_autograd(x if B > 1 else x[0], torch.as_tensor(ell).cuda(), n_tr, cn, tn, 0.3, sparse)
    if B == 1:
        cov = cov[None]
    if sparse:
        wc = w
    else:
        wc = torch.randn(B, n * n_ell, n * n_ell, generator=gen, dtype=torch.float64).cuda()  # off-diagonals: no effect
        i = torch.arange(n_ell, device="cuda")
        wc.view(B, n, n_ell, n, n_ell)[:, :, i, :, i] = w.permute(3, 0, 1, 2)
    got, = torch.autograd.grad((cov * wc).sum(), x, retain_graph=True)
    assert float((got - ref).abs().max()) < 1e-13 * float(ref.abs().max())
    graph, = torch.autograd.grad((cov * wc.requires_grad_(True)).sum(), x, create_graph=True)
    assert graph.requires_grad
    assert float((graph - ref).abs().max()) < 1e-13 * float(ref.abs().max())


@pytest.mark.parametrize("logdet", [True, False])
def test_loglike_gradient_in_a_batch_of_sparse_covariances(logdet):
    gen = torch.Generator().manual_seed(4)
    B, n, nl = 3, 5, 7
    a = torch.randn(B, nl, n, n, generator=gen, dtype=torch.float64)
    blocks = (a @ a.transpose(-1, -2) + n * torch.eye(n, dtype=torch.float64)).cuda()
    data, mu = (torch.randn(B, n * nl, generator=gen, dtype=torch.float64).cuda() for _ in range(2))
    go = torch.randn(B, generator=gen, dtype=torch.float64).cuda()
    C = blocks.permute(0, 2, 3, 1).contiguous().requires_grad_(True)
    out = jc.likelihood.gaussian_log_likelihood(data, mu, C, include_logdet=logdet)
    got, = torch.autograd.grad((out * go).sum(), C)
    Cr = blocks.permute(0, 2, 3, 1).contiguous().requires_grad_(True)
    bl, r = Cr.permute(0, 3, 1, 2), (mu - data).reshape(B, n, nl).transpose(1, 2)
    q = (r * torch.linalg.solve(bl, r)).sum((1, 2))
    ref = -0.5 * (q - torch.linalg.slogdet(bl)[1].sum(1)) if logdet else -0.5 * q
    want, = torch.autograd.grad((ref * go).sum(), Cr)
    assert float((got - want).abs().max()) < 1e-12 * float(want.abs().max())
