"""Backward passes under vectorised Jacobians, forward mode and create_graph: the
log-likelihood's and the covariance's gradients carry batches of cotangents and
their tangents on.  The kernels' calls are replaced by torch forms here (CPU);
``test_gpu_backward_transforms.py`` runs the library's."""
import numpy as np
import pytest
import torch
from torch.autograd import forward_ad as fw

from jax_cosmo_gb300 import _lib, autodiff, likelihood

N_CLS, N_ELL, B = 3, 4, 3


@pytest.fixture(autouse=True)
def torch_forms(monkeypatch):
    """libjcg's calls as torch operations on the tensors behind their pointers."""
    seen = {}

    def ptr(t):
        if t is None:
            return None
        t.data_ptr()  # raises for a tensor without storage
        seen[id(t)] = t.detach()  # a kernel sees values
        return id(t)

    def core(data, mu, C, sparse, n_cls, n_ell, include_logdet, alpha=None):
        blocks, r = C.permute(0, 3, 1, 2), (mu - data).reshape(-1, n_cls, n_ell).transpose(1, 2)
        x = torch.linalg.solve(blocks, r)
        alpha.copy_(x.transpose(1, 2).reshape(mu.shape))
        q = (r * x).sum((1, 2)) - (torch.linalg.slogdet(blocks)[1].sum(-1) if include_logdet else 0.0)
        return -0.5 * q, torch.zeros(len(mu), dtype=torch.int32)

    def call(name, *args):
        assert name == "jcg_gaussian_loglike_cov_grad"
        a, inv, go, out = (seen.get(args[i]) for i in (0, 1, 2, 6))
        a = a.reshape(B, N_CLS, N_ELL)
        v = torch.einsum("bpl,bql->bpql", a, a) + (0.0 if inv is None else inv)
        out.copy_(0.5 * go[:, None, None, None] * v)

    monkeypatch.setattr(_lib, "ptr", ptr)
    monkeypatch.setattr(_lib, "call", call)
    monkeypatch.setattr(_lib, "stream_of", lambda device: None)
    monkeypatch.setattr(likelihood, "_loglike_core", core)
    monkeypatch.setattr(autodiff, "_sparse_inv_batched",
                        lambda s: torch.linalg.inv(s.permute(0, 3, 1, 2)).permute(0, 2, 3, 1).contiguous())


def inputs():
    g = torch.Generator().manual_seed(1)
    a = torch.randn(B, N_ELL, N_CLS, N_CLS, dtype=torch.float64, generator=g)
    C = (a @ a.transpose(-1, -2) + N_CLS * torch.eye(N_CLS, dtype=torch.float64)).permute(0, 2, 3, 1).contiguous()
    data, mu = (torch.randn(B, N_CLS * N_ELL, dtype=torch.float64, generator=g) for _ in range(2))
    return data, mu, C


def loglike(data, mu, C, logdet):
    return autodiff.loglike_autograd(data, mu, C, logdet, True, N_CLS, N_ELL)


@pytest.mark.parametrize("logdet", [True, False])
def test_vectorised_jacobian_in_the_covariance(logdet):
    data, mu, C = inputs()
    f = lambda c: loglike(data, mu, c, logdet)  # noqa: E731
    one = torch.autograd.functional.jacobian(f, C)
    assert torch.allclose(torch.autograd.functional.jacobian(f, C, vectorize=True), one, rtol=1e-13, atol=0)
    x = C.clone().requires_grad_(True)
    (b,) = torch.autograd.grad(f(x), x, torch.eye(B, dtype=torch.float64), is_grads_batched=True)
    assert torch.allclose(b, one, rtol=1e-13, atol=0)


def test_a_cotangents_forward_tangent_goes_on():
    data, mu, C = inputs()
    x = C.clone().requires_grad_(True)
    go, dgo = torch.tensor([0.3, -1.0, 2.0], dtype=torch.float64), torch.tensor([1.0, 0.5, -0.2], dtype=torch.float64)
    ll = loglike(data, mu, x, True)
    (want,) = torch.autograd.grad(ll, x, dgo, retain_graph=True)
    (value,) = torch.autograd.grad(ll, x, go, retain_graph=True)
    with fw.dual_level():
        (g,) = torch.autograd.grad(ll, x, fw.make_dual(go, dgo))
        p, t = fw.unpack_dual(g)
        assert t is not None and torch.allclose(t, want, rtol=1e-13, atol=0)
        assert torch.allclose(p, value, rtol=1e-13, atol=0)


def test_covariance_cotangents_forward_tangent_goes_on(monkeypatch):
    def call(name, *args):
        pytest.fail("a cotangent with a tangent went to the kernel")

    monkeypatch.setattr(_lib, "call", call)
    from jax_cosmo_gb300 import angular_cl

    n_tr, n_cls = 2, 3
    monkeypatch.setattr(angular_cl, "_covariance",
                        lambda ell, n, cl, cn, tn, f, sparse: torch.zeros(n_cls, n_cls, N_ELL, dtype=torch.float64))
    ell = torch.tensor(np.geomspace(10.0, 100.0, N_ELL))
    cl = torch.rand(n_cls, N_ELL, dtype=torch.float64, generator=torch.Generator().manual_seed(2), requires_grad=True)
    cov = autodiff.covariance_autograd(cl, ell, n_tr, None, None, 0.3, True)
    w, dw = (torch.randn(n_cls, n_cls, N_ELL, dtype=torch.float64, generator=torch.Generator().manual_seed(s)) for s in (3, 4))
    (want,) = torch.autograd.grad(cov, cl, dw.requires_grad_(True), retain_graph=True, create_graph=True)
    with fw.dual_level():
        (g,) = torch.autograd.grad(cov, cl, fw.make_dual(w, dw.detach()))
        t = fw.unpack_dual(g).tangent
        assert t is not None and torch.allclose(t, want.detach(), rtol=1e-13, atol=0)
