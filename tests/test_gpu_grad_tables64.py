"""The float64 Jacobian's tables (background, growth, sigma8, P(k), sigma^2(R)
with tangents) over the options that take another branch there: both transfer
types, curvature with w0 and wa, a small Omega_b, and the
number of cosmologies up to and past the scalars' half-warp form.

Tolerance: the tables hold sums of at most 257 positive terms and products of
about 100 factors, a few 1e-14; the Limber sums and the oracle's autograd add as
much, and a column's entries cancel by a factor of 100 at most: 1e-11 of the
column's largest entry.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import functools  # noqa: E402

import jax_cosmo_gb300 as jc  # noqa: E402
from oracle import jc_oracle as O  # noqa: E402

ELL = np.geomspace(10, 3000, 7)


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def probes():
    nz = [jc.redshift.smail_nz(1.0, 2.0, z, gals_per_arcmin2=10.0, zmax=4.0) for z in (0.5, 1.0)]
    return [jc.probes.WeakLensing(nz[:1], sigma_e=0.26), jc.probes.NumberCounts(nz[1:], jc.bias.constant_linear_bias(1.2))]


def oracle_probes():
    nz = [O.Smail(1.0, 2.0, z, 4.0, 10.0) for z in (0.5, 1.0)]
    return [O.Probe("wl", nz[:1], sigma_e=0.26), O.Probe("nc", nz[1:], bias=1.2)]


def cosmo(rows):
    rows = torch.tensor(np.atleast_2d(rows), dtype=torch.float64, device="cuda")
    return jc.Cosmology(*[rows[:, i] for i in range(8)])


@pytest.mark.parametrize("transfer", ["eisenhu_osc", "eisenhu"])
@pytest.mark.parametrize("row", [
    [0.2589, 0.0486, 0.6774, 0.9667, 0.8159, 0.0, -1.0, 0.0],
    [0.31, 0.045, 0.66, 0.98, 0.72, 0.02, -0.85, 0.15],
    [0.25, 0.004, 0.7, 0.9, 1.0, -0.02, -1.3, -0.3],
])
def test_jacobian_vs_oracle(row, transfer):
    def f(v):
        cs = O.Cosmo.from_vector(v)
        cs.transfer = transfer
        return O.angular_cl(cs, ELL, oracle_probes(), n_limber=128)

    v0 = torch.tensor(row, dtype=torch.float64)
    ref = torch.autograd.functional.jacobian(f, v0)
    tf = functools.partial(jc.transfer.Eisenstein_Hu, type=transfer)
    _, jac = jc.autodiff.angular_cl_jacobian(cosmo(row), ELL, probes(), 128, "fp64", transfer_fn=tf)
    err = (jac[0].cpu() - ref).abs().amax((0, 1)) / ref.abs().amax((0, 1))
    assert float(err.max()) < 1e-11, err


@pytest.mark.parametrize("B", [2, 129])
def test_a_batch_equals_its_single_cosmologies(B):
    """Up to 128 cosmologies only the order of the Limber sum over a differs
    (1e-13); past it the scalars' kernel changes and with it the rounding of the Eisenstein-Hu scalars: 1e-11."""
    rng = np.random.default_rng(3)
    lo = np.array([0.2, 0.04, 0.6, 0.9, 0.6, -0.02, -1.3, -0.3])
    rows = lo + np.array([0.15, 0.02, 0.2, 0.1, 0.4, 0.04, 0.6, 0.6]) * rng.random((B, 8))
    _, jb = jc.autodiff.angular_cl_jacobian(cosmo(rows), ELL, probes(), 128)
    for i in (0, B - 1):
        _, j1 = jc.autodiff.angular_cl_jacobian(cosmo(rows[i]), ELL, probes(), 128)
        err = (jb[i] - j1[0]).abs().amax((0, 1)) / j1[0].abs().amax((0, 1))
        assert float(err.max()) <= (1e-11 if B > 128 else 1e-13)
