"""The dense covariance's rows at odd and even lengths (16-byte stores from
either alignment), one and several cosmologies, against the sparse form: the
same elements bit for bit, zeros elsewhere."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import jax_cosmo_gb300 as jc  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


@pytest.mark.parametrize("n_tr,n_ell,B", [(1, 2, 1), (2, 5, 1), (2, 5, 3), (3, 300, 1), (5, 17, 2), (4, 8, 1)])
@pytest.mark.parametrize("with_noise", [False, True])
def test_dense_equals_sparse(n_tr, n_ell, B, with_noise):
    rng = np.random.default_rng(n_tr * 100 + n_ell)
    n_cls = n_tr * (n_tr + 1) // 2
    nz = [jc.redshift.smail_nz(1.0, 2.0, 0.5 + 0.1 * i, gals_per_arcmin2=10.0, zmax=4.0) for i in range(n_tr)]
    probes = [jc.probes.WeakLensing(nz, sigma_e=0.26)]
    ell = np.sort(rng.uniform(10, 3000, n_ell))
    cl = torch.tensor(rng.uniform(1e-9, 1e-8, (B, n_cls, n_ell)), device="cuda")
    noise = torch.tensor(rng.uniform(1e-10, 1e-9, (n_cls, n_ell)), device="cuda") if with_noise else torch.zeros(
        n_cls, n_ell, dtype=torch.float64, device="cuda")
    sp = jc.cl.gaussian_cl_covariance(ell, probes, cl, noise, sparse=True)
    torch.empty(cl.numel() * 64, dtype=torch.float64, device="cuda").fill_(7.0)  # what the buffer held before
    de = jc.cl.gaussian_cl_covariance(ell, probes, cl, noise, sparse=False)
    want = torch.zeros(B, n_cls, n_ell, n_cls, n_ell, dtype=torch.float64, device="cuda")
    i = torch.arange(n_ell, device="cuda")
    want[:, :, i, :, i] = sp.permute(3, 0, 1, 2)
    assert torch.equal(de, want.reshape(B, n_cls * n_ell, n_cls * n_ell))
