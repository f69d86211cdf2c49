"""The float64 gradient's radial kernels where their loops can go wrong: 1, 3, 4 and
7 lensing bins (passes of three), two lensing groups with a single plane and
alignment terms, n(z) so near that chi is below 1 (its clip), node counts of one
CTA and of several with one node left over.

Tolerance: a kernel's tangent is the difference of sums of 257 positive products
of 2^-47 each, ten times larger than itself at worst; the Limber integral as in
its own test: 2e-12 of each spectrum's and parameter's largest entry.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import jax_cosmo_gb300 as jc  # noqa: E402
from oracle import jc_oracle as O  # noqa: E402

ROW = [0.27, 0.047, 0.69, 0.96, 0.81, 0.01, -0.95, 0.1]
ELL = np.array([12.0, 150.0, 2200.0])


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def check(p, o, n_limber):
    def f(v):
        return O.angular_cl(O.Cosmo.from_vector(v), ELL, o, n_limber=n_limber)

    v = torch.tensor(ROW, dtype=torch.float64)
    ref = torch.autograd.functional.jacobian(f, v, strategy="forward-mode", vectorize=True)
    names = ["Omega_c", "Omega_b", "h", "n_s", "sigma8", "Omega_k", "w0", "wa"]
    _, jac = jc.autodiff.angular_cl_jacobian(jc.Cosmology(**dict(zip(names, ROW))), ELL, p, n_limber)
    err = (jac.cpu() - ref).abs().amax(-2) / ref.abs().amax(-2)
    scale = ref.abs().amax((0, 1)) / ref.abs().amax((0, 1)).max()
    assert float((err * torch.clamp(scale, 0.01, 1.0)).max()) < 2e-12, err.max()


@pytest.mark.parametrize("n_wl,zmax,n_limber", [(1, 4.0, 8), (3, 10.0, 32), (4, 3.0, 64), (7, 4.0, 40)])
def test_bins_and_nodes(n_wl, zmax, n_limber):
    z0 = np.linspace(0.3, 1.1, n_wl)
    p = [jc.probes.WeakLensing([jc.redshift.smail_nz(1.0, 2.0, float(z), zmax=zmax) for z in z0], sigma_e=0.26,
                               multiplicative_bias=0.02)]
    o = [O.Probe("wl", [O.Smail(1.0, 2.0, float(z), zmax, 1.0) for z in z0], sigma_e=0.26, m=0.02)]
    check(p, o, n_limber)


def test_groups_planes_and_alignment():
    nz = [jc.redshift.smail_nz(1.0, 2.0, z, zmax=zm) for z, zm in ((0.5, 3.0), (0.9, 6.0))]
    oz = [O.Smail(1.0, 2.0, z, zm, 1.0) for z, zm in ((0.5, 3.0), (0.9, 6.0))]
    p = [jc.probes.WeakLensing(nz[:1], ia_bias=jc.bias.des_y1_ia_bias(0.8, 1.3, 0.62)),
         jc.probes.WeakLensing([nz[1], jc.redshift.delta_nz(1.1, zmax=6.0)]),
         jc.probes.NumberCounts(nz[:1], jc.bias.inverse_growth_linear_bias(1.3))]
    o = [O.Probe("wl", oz[:1], ia=("desy1", 0.8, 1.3, 0.62)), O.Probe("wl", [oz[1], O.Delta(1.1, 6.0)]),
         O.Probe("nc", oz[:1], bias=("invg", 1.3))]
    check(p, o, 96)


def test_chi_below_one():
    """zmax of 5e-4: comoving distances of 0 to 1.5 Mpc/h, k of 10 to 10^4."""
    p = [jc.probes.WeakLensing([jc.redshift.smail_nz(1.0, 2.0, 2e-4, zmax=5e-4)], sigma_e=0.26)]
    check(p, [O.Probe("wl", [O.Smail(1.0, 2.0, 2e-4, 5e-4, 1.0)], sigma_e=0.26)], 16)


@pytest.mark.parametrize("gamma_dir", [2, 3, 4])
def test_gamma_in_a_direction_without_background(gamma_dir):
    """d C_ell / d gamma does not depend on the direction that carries it: in those of h,
    n_s and sigma_8 the kernels' tangents are otherwise left out.  Biases with the
    growth factor give the kernels a tangent in gamma."""
    from jax_cosmo_gb300 import _lib
    from jax_cosmo_gb300.autodiff import jacobian_device

    nz = [jc.redshift.smail_nz(1.0, 2.0, z, zmax=4.0) for z in (0.5, 0.9)]
    p = [jc.probes.WeakLensing(nz[:1], ia_bias=jc.bias.inverse_growth_linear_bias(0.7)),
         jc.probes.NumberCounts(nz[1:], jc.bias.inverse_growth_linear_bias(1.3))]
    params = torch.tensor([ROW + [0.55]], dtype=torch.float64, device="cuda")
    _, a = jacobian_device(params, ELL, p, 64, "fp64", _lib.GROWTH_GAMMA, gamma_dir=0)
    _, b = jacobian_device(params, ELL, p, 64, "fp64", _lib.GROWTH_GAMMA, gamma_dir=gamma_dir)
    ref, got = a[0, ..., 0], b[0, ..., gamma_dir]
    assert float(((got - ref).abs().amax(-1) / ref.abs().amax(-1)).max()) < 2e-12
