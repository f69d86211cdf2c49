"""Pointwise queries over point counts where their CTAs change: one or two points a
CTA, up to 256, and several cosmologies across a CTA; the background functions a
thread per point.  A point's value does not depend on the others of its call: it is
compared bit for bit with the call of that point alone, and some with the oracle
(1e-12: each is some 100 float64 operations)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import jax_cosmo_gb300 as jc  # noqa: E402
from oracle import jc_oracle as O  # noqa: E402

NAMES = ["Omega_c", "Omega_b", "h", "n_s", "sigma8", "Omega_k", "w0", "wa"]
ROW = [0.27, 0.047, 0.69, 0.96, 0.81, 0.01, -0.95, 0.1]


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def rows(n):
    return np.array(ROW) * (1.0 + 0.03 * np.random.default_rng(n).standard_normal((n, 8)))


def cosmo(r):
    return jc.Cosmology(**{n: torch.tensor(r[:, i], device="cuda") for i, n in enumerate(NAMES)})


@pytest.mark.parametrize("n_cosmo,n", [(1, 1), (1, 2), (1, 305), (3, 33), (2, 1300), (70, 1200)])
def test_nonlinear_power(n_cosmo, n):
    rng = np.random.default_rng(n)
    k, a, r = 10.0 ** rng.uniform(-4, 1, n), rng.uniform(0.2, 1.0, n), rows(n_cosmo)
    out = jc.power.nonlinear_matter_power(cosmo(r), k, a).cpu()
    assert out.shape == (n_cosmo, n) and bool(torch.isfinite(out).all())
    for i, j in {(0, 0), (n_cosmo - 1, n - 1), (n_cosmo // 2, n // 2), (n_cosmo // 3, n // 3)}:
        one = jc.power.nonlinear_matter_power(cosmo(r[i:i + 1]), k[j:j + 1], a[j:j + 1]).cpu()
        assert float(one[0, 0]) == float(out[i, j])
        ref = O.halofit_nodes(O.Cosmo.from_vector(list(r[i])), torch.tensor([[k[j]]]), torch.tensor([a[j]]))
        assert abs(float(one[0, 0]) / float(ref.reshape(-1)[0]) - 1.0) < 1e-12


@pytest.mark.parametrize("n", [1, 33, 20000])
def test_background_and_linear_power(n):
    rng = np.random.default_rng(n)
    a, k, r = rng.uniform(0.05, 1.0, n), 10.0 ** rng.uniform(-4, 1, n), rows(2)
    c, one = cosmo(r), cosmo(r[1:])
    for f in (jc.background.radial_comoving_distance, jc.background.growth_factor, jc.background.growth_rate,
              jc.background.H, jc.background.dchioverda, jc.background.transverse_comoving_distance):
        v = f(c, a).cpu()
        assert float(v[1, n - 1]) == float(f(one, a[n - 1:]).cpu()[0, 0])
        assert float(v[1, n // 2]) == float(f(one, a[n // 2:n // 2 + 1]).cpu()[0, 0])
    v = jc.power.linear_matter_power(c, k, a).cpu()
    assert float(v[1, n - 1]) == float(jc.power.linear_matter_power(one, k[n - 1:], a[n - 1:]).cpu()[0, 0])
    chi = jc.background.radial_comoving_distance(c, a)
    back = jc.background.a_of_chi(c, chi[0].cpu().numpy()).cpu()
    assert back.shape[-1] == n and bool(torch.isfinite(back).all())
