"""The float64 method's Limber integral at the sizes where its tiling can go
wrong: the a nodes in blocks of up to 72 (one node left over, one block, more
blocks than a cluster has CTAs), ell tiles of 1, odd and more than 128 ell, 1 to
136 spectra, and the blocks that leave the range of float pairs.

Tolerance: a node's value is some 60 pair operations of 2^-47 each at worst,
twice that for the square of the transfer function: 1e-12 of the oracle.
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


def probes(n_wl, n_nc, zmax=4.0):
    z0 = np.linspace(0.3, 1.2, max(n_wl, n_nc, 1))
    nz = [jc.redshift.smail_nz(1.0, 2.0, float(z), gals_per_arcmin2=10.0, zmax=zmax) for z in z0]
    onz = [O.Smail(1.0, 2.0, float(z), zmax, 10.0) for z in z0]
    p, o = [], []
    if n_wl:
        p.append(jc.probes.WeakLensing(nz[:n_wl], sigma_e=0.26))
        o.append(O.Probe("wl", onz[:n_wl], sigma_e=0.26))
    if n_nc:
        p.append(jc.probes.NumberCounts(nz[:n_nc], jc.bias.constant_linear_bias(1.2)))
        o.append(O.Probe("nc", onz[:n_nc], bias=1.2))
    return p, o


def batch(rows):
    return jc.Cosmology(*[torch.tensor(np.asarray(rows)[:, i], dtype=torch.float64, device="cuda") for i in range(8)])


@pytest.mark.parametrize("n_limber,n_ell,n_wl,n_nc", [
    (2, 1, 1, 0), (70, 1, 1, 0), (72, 33, 1, 1), (142, 129, 0, 1), (144, 7, 2, 1), (576, 131, 1, 0),
    (1024, 5, 1, 1), (256, 9, 8, 8),
])
def test_sizes_vs_oracle(n_limber, n_ell, n_wl, n_nc):
    p, o = probes(n_wl, n_nc)
    ell = np.logspace(1, 3.5, n_ell) if n_ell > 1 else np.array([57.3])
    cl = jc.cl.angular_cl(batch([ROW]), ell, p, n_limber=n_limber)[0].cpu()
    ref = O.angular_cl(O.Cosmo.from_vector(ROW), ell, o, n_limber=n_limber)
    assert float(((cl - ref) / ref).abs().max()) < 1e-12


@pytest.mark.parametrize("n_limber", [256, 512, 1024])
def test_one_cosmology_equals_its_row_of_a_large_batch(n_limber):
    """Clusters (one cosmology) and one CTA per tile (many) make the same sums."""
    p, _ = probes(2, 1)
    ell = np.logspace(1, 3.5, 21)
    rng = np.random.default_rng(3)
    rows = np.array([ROW] * 700) * (1 + 0.01 * rng.uniform(-1, 1, (700, 8)))
    big = jc.cl.angular_cl(batch(rows), ell, p, n_limber=n_limber)
    for b in (0, 333, 699):
        assert torch.equal(big[b], jc.cl.angular_cl(batch(rows[b:b + 1]), ell, p, n_limber=n_limber)[0])


def test_outside_the_pairs_range():
    """ell of 10^7 and more, a spectrum's weights of 1e-200, and a non-finite cosmology in a batch."""
    p, o = probes(1, 1)
    ell = np.array([30.0, 3e4, 2e7])
    cl = jc.cl.angular_cl(batch([ROW]), ell, p, n_limber=128)[0].cpu()
    ref = O.angular_cl(O.Cosmo.from_vector(ROW), ell, o, n_limber=128)
    assert float(((cl - ref) / ref).abs().max()) < 1e-9  # sin(k s) at 10^9 radians: float64 argument rounding
    ell = np.array([30.0, 300.0])
    nz = [jc.redshift.smail_nz(1.0, 2.0, z, zmax=4.0) for z in (0.02, 1.0)]
    onz = [O.Smail(1.0, 2.0, z, 4.0, 1.0) for z in (0.02, 1.0)]
    cl = jc.cl.angular_cl(batch([ROW]), ell, [jc.probes.NumberCounts(nz, jc.bias.constant_linear_bias(1.0))], n_limber=128)[0].cpu()
    ref = O.angular_cl(O.Cosmo.from_vector(ROW), ell, [O.Probe("nc", onz, bias=1.0)], n_limber=128)
    assert float(((cl - ref) / ref).abs().max()) < 1e-12
    bad = np.array([ROW, ROW, ROW])
    bad[1, 2] = np.nan
    got = jc.cl.angular_cl(batch(bad), ell, p, n_limber=128)
    one = jc.cl.angular_cl(batch([ROW]), ell, p, n_limber=128)
    assert torch.isnan(got[1]).all() and torch.equal(got[0], one[0]) and torch.equal(got[2], one[0])
