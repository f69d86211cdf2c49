"""Per-ell block inverse and log-likelihood at the sizes where the number of
registers per thread, the threads per CTA or the back substitution's lanes
change, against torch in float64.

Blocks are A = Q diag(1 .. 30) Q^T-like, condition number about 30: n = 160
eliminations of 2^-53 each, times the condition number, stay below 1e-12.
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


def spd(n, nd, seed, B=1):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(B, nd, n, n, dtype=torch.float64, device="cuda", generator=g)
    q, _ = torch.linalg.qr(x)
    lam = torch.linspace(1.0, 30.0, n, dtype=torch.float64, device="cuda")
    a = (q * lam) @ q.transpose(-1, -2)
    a = 0.5 * (a + a.transpose(-1, -2))
    return a.permute(0, 2, 3, 1).contiguous()  # [B, n, n, nd]


def inv_ref(a):
    return torch.linalg.inv(a.permute(0, 3, 1, 2)).permute(0, 2, 3, 1)


SIZES = [1, 2, 3, 14, 15, 16, 30, 31, 32, 33, 55, 57, 58, 59, 60, 94, 95, 96, 136, 159, 160]


@pytest.mark.parametrize("n", SIZES)
def test_inverse_of_symmetric_blocks(n):
    a = spd(n, 3, n, B=2)
    got = jc.sparse.inv_batched(a)
    ref = inv_ref(a)
    assert float((got - ref).norm() / ref.norm()) < TOL
    assert torch.equal(got, got.transpose(1, 2))


@pytest.mark.parametrize("n", [2, 15, 55, 160])
def test_blocks_that_are_not_symmetric_or_not_positive(n):
    a = spd(n, 4, 7 * n)
    a[0, 0, 1, 1] += 0.25                      # not symmetric
    a[0, :, :, 2] -= 40.0 * torch.eye(n, dtype=a.dtype, device=a.device)   # negative definite
    a[0, :, :, 3] = torch.flip(torch.eye(n, dtype=a.dtype, device=a.device), [0])  # symmetric, zero pivots
    got, ref = jc.sparse.inv(a[0]), inv_ref(a)[0]
    for l in range(4):
        assert float((got[..., l] - ref[..., l]).norm() / ref[..., l].norm()) < 10 * TOL, l


def test_inverse_passes_non_finite_values_on():
    a = spd(6, 2, 1)[0].contiguous()
    a[2, 2, 1] = float("nan")
    got = jc.sparse.inv(a)
    assert torch.isfinite(got[..., 0]).all() and torch.isnan(got[..., 1]).any()


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dense", [False, True])
def test_loglike_and_its_gradients(n, dense):
    nd, B = 3, 2
    if dense and n > 60:
        pytest.skip("the dense form shares the kernel; its matrix would be large")
    c = spd(n, nd, 100 + n, B)
    g = torch.Generator(device="cuda").manual_seed(n)
    mu = torch.randn(B, n * nd, dtype=torch.float64, device="cuda", generator=g)
    data = torch.randn(n * nd, dtype=torch.float64, device="cuda", generator=g)
    blocks = c.permute(0, 3, 1, 2)
    r = (mu - data).reshape(B, n, nd).permute(0, 2, 1)[..., None]
    al = torch.linalg.solve(blocks, r)
    ref = -0.5 * ((r * al).sum((1, 2, 3)) - torch.linalg.slogdet(blocks)[1].sum(-1))
    C = c
    if dense:
        C = torch.zeros(B, n, nd, n, nd, dtype=torch.float64, device="cuda")
        i = torch.arange(nd, device="cuda")
        C[:, :, i, :, i] = c.permute(3, 0, 1, 2)
        C = C.reshape(B, n * nd, n * nd)
        C._jcg_n_ell = nd
    m = mu.clone().requires_grad_(True)
    ll = jc.likelihood.gaussian_log_likelihood(data, m, C)
    assert float(((ll.detach() - ref) / ref).abs().max()) < TOL
    (dm,) = torch.autograd.grad(ll.sum(), m)
    want = -al[..., 0].permute(0, 2, 1).reshape(B, n * nd)
    assert float((dm - want).norm() / want.norm()) < TOL


def test_loglike_flags_a_block_that_is_not_positive():
    c = spd(7, 3, 5, 2)
    c[1, :, :, 2] = -c[1, :, :, 2]
    mu = torch.zeros(2, 21, dtype=torch.float64, device="cuda")
    ll = jc.likelihood.gaussian_log_likelihood(torch.ones(21, dtype=torch.float64, device="cuda"), mu, c)
    assert torch.isfinite(ll[0]) and torch.isnan(ll[1])
