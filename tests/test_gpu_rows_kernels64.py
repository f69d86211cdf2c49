"""The float64 method's halofit rows and radial kernels at the sizes and inputs
where their tiling and their pair arithmetic can go wrong.

Tolerances: a radial kernel's integral is a sum of positive terms of some ten
pair operations (2^-47 each at worst): 1e-13, times the cancellation of chi' -
chi where the node is far above the bin, for which the oracle's float64 itself
leaves 1e-12 of the kernel.  C_ell: 1e-12 (as for the Limber integral).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import jax_cosmo_gb300 as jc  # noqa: E402
from oracle import jc_oracle as O  # noqa: E402

ROW = [0.27, 0.047, 0.69, 0.96, 0.81, 0.01, -0.95, 0.1]


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def batch(rows):
    return jc.Cosmology(*[torch.tensor(np.asarray(rows)[:, i], dtype=torch.float64, device="cuda") for i in range(8)])


def smail(z0, zmax=4.0):
    return jc.redshift.smail_nz(1.0, 2.0, z0, gals_per_arcmin2=10.0, zmax=zmax), O.Smail(1.0, 2.0, z0, zmax, 10.0)


@pytest.mark.parametrize("B", [1, 95, 96, 130])
@pytest.mark.parametrize("z0s", [(0.5,), (0.3, 0.6, 0.9, 1.2, 1.5, 1.8, 2.1, 2.4), tuple(0.3 + 0.15 * i for i in range(9))])
def test_lensing_kernels_vs_oracle(B, z0s):
    """Both forms of the kernel stage (fewer than 96 cosmologies, more; 1, 8 and 9 bins)."""
    z = np.concatenate([[1e-3], np.linspace(0.02, 3.9, 38)])
    bins = [smail(float(v)) for v in z0s]
    p = jc.probes.WeakLensing([b[0] for b in bins], sigma_e=0.26, multiplicative_bias=0.02)
    rows = np.array([ROW] * B)
    rows[:, 0] += 0.001 * np.arange(B)
    got = p.kernel(batch(rows), z, 20.0).cpu()
    for b in (0, B - 1):
        ref = O.probe_kernel(O.Cosmo.from_vector(rows[b]), O.Probe("wl", [v[1] for v in bins], sigma_e=0.26, m=0.02),
                             torch.as_tensor(z), 20.0)
        assert float(((got[b] - ref) / ref).abs().max()) < 1e-11
        assert float((got[b] - ref).norm() / ref.norm()) < 1e-13


@pytest.mark.parametrize("B", [1, 100])
def test_ragged_grids_special_bias_and_planes(B):
    """Two lensing grids, NLA, inverse-growth bias and a single-plane bin; a batch
    row equals the cosmology alone bit for bit."""
    nz = [smail(0.4, 3.0), smail(0.9, 4.0)]
    probes = [jc.probes.WeakLensing([nz[0][0]], ia_bias=jc.bias.des_y1_ia_bias(0.8, 1.3, 0.62)),
              jc.probes.WeakLensing([nz[1][0], jc.redshift.delta_nz(1.1, zmax=4.0)]),
              jc.probes.NumberCounts([nz[1][0]], jc.bias.inverse_growth_linear_bias(1.1))]
    oprobes = [O.Probe("wl", [nz[0][1]], ia=("desy1", 0.8, 1.3, 0.62)), O.Probe("wl", [nz[1][1], O.Delta(1.1, 4.0)]),
               O.Probe("nc", [nz[1][1]], bias=("invg", 1.1))]
    ell = np.logspace(1, 3, 9)
    rows = np.array([ROW] * B)
    rows[:, 4] += 0.002 * np.arange(B)
    cl = jc.cl.angular_cl(batch(rows), ell, probes, n_limber=130)
    ref = O.angular_cl(O.Cosmo.from_vector(rows[B - 1]), ell, oprobes, n_limber=130)
    assert float((cl[B - 1].cpu() - ref).norm() / ref.norm()) < 1e-12
    assert torch.equal(cl[B - 1], jc.cl.angular_cl(batch(rows[B - 1:]), ell, probes, n_limber=130)[0])


def test_kernels_do_not_depend_on_the_batch():
    bins = [smail(float(v))[0] for v in (0.4, 0.8, 1.2)]
    p = [jc.probes.WeakLensing(bins), jc.probes.NumberCounts(bins, jc.bias.constant_linear_bias(1.3))]
    rows = np.array([ROW] * 300)
    rows[:, 3] -= 0.0002 * np.arange(300)
    ell = np.logspace(1, 3, 6)
    big = jc.cl.angular_cl(batch(rows), ell, p)
    for B, b in ((1, 0), (95, 140), (96, 33)):
        part = jc.cl.angular_cl(batch(rows[b:b + B]), ell, p)
        assert torch.equal(part, big[b:b + B])


def test_halofit_scale_extremes_vs_oracle():
    """Amplitudes that move the non-linear scale to both ends of its table, and
    the k_nl clip; every model's coefficients."""
    nz = smail(0.8)
    ell = np.logspace(1, 3, 5)
    for s8 in (0.02, 0.3, 3.0):
        row = list(ROW)
        row[4] = s8
        for nl, name in ((jc.power.halofit, "takahashi2012"), (jc.power.linear_matter_power, "linear")):
            cl = jc.cl.angular_cl(batch([row]), ell, [jc.probes.WeakLensing([nz[0]])], nonlinear_fn=nl, n_limber=66)
            ref = O.angular_cl(O.Cosmo.from_vector(row), ell, [O.Probe("wl", [nz[1]])], n_limber=66, nonlinear=name)
            assert float(((cl[0].cpu() - ref) / ref).abs().max()) < 1e-11, (s8, name)
