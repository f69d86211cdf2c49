"""The Eisenstein-Hu scalars of the float64 gradient have two forms: half a warp per
(cosmology, direction) up to 128 cosmologies and a thread from there on.  Both use
the same formulas: C_ell and the Jacobian of a cosmology agree across the change to
the rounding of quotients taken in another order.

Baryon fractions of 0.3 to 0.7, where P(k) is made of the baryons' terms.
Tolerance: ten roundings of 2^-53 in a scalar, twice that for T^2, and as much for
the sums over a where they are associated otherwise: 4e-15 of a C_ell; a tangent
column's entries cancel by a factor of five: 2e-14 of its largest entry."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import jax_cosmo_gb300 as jc  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


@pytest.mark.parametrize("matter", [(0.08, 0.08, 0.10, 0.10), (0.4, 0.3, 0.3, 0.3)])
def test_across_the_change_of_form(matter):
    rng = np.random.default_rng(5)
    lo = np.array([matter[0], matter[2], 0.6, 0.9, 0.6, 0.0, -1.2, -0.2])
    rows = lo + np.array([matter[1], matter[3], 0.2, 0.1, 0.4, 0.0, 0.4, 0.4]) * rng.random((129, 8))
    nz = [jc.redshift.smail_nz(1.0, 2.0, z, gals_per_arcmin2=10.0, zmax=4.0) for z in (0.5, 1.0)]
    probes = [jc.probes.WeakLensing(nz[:1], sigma_e=0.26), jc.probes.NumberCounts(nz[1:], jc.bias.constant_linear_bias(1.2))]

    def jac(r):
        t = torch.tensor(r, dtype=torch.float64, device="cuda")
        return jc.autodiff.angular_cl_jacobian(jc.Cosmology(*[t[:, i] for i in range(8)]), np.geomspace(10, 3000, 9), probes, 128)

    few, many = jac(rows[:128]), jac(rows)
    assert float(((many[0][:128] - few[0]) / few[0]).abs().max()) < 4e-15
    err = (many[1][:128] - few[1]).abs().amax((1, 2)) / few[1].abs().amax((1, 2))
    assert float(err.max()) < 2e-14
