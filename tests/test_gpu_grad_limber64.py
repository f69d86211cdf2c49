"""The float64 Jacobian's Limber integral in float pairs at the sizes where its
tiling can go wrong: a nodes in chunks of up to 16 (one node, one left over, one
chunk, several splits), ell tiles of 1, odd and 32, 1 to 136 spectra, all operator
points, ragged batches, and the cosmologies that leave the range of float pairs
(recomputed in float64).

Tolerance: a node's tangent is a sum of some 20 terms, ten times larger than
itself at worst, of 2^-47 each: 2e-12 of the column's largest entry with the
oracle's own rounding; 1e-9 at arguments of 10^9 radians.
"""
import functools

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


def oracle(row, ell, o, n_limber, transfer="eisenhu_osc", nonlinear="takahashi2012"):
    def f(v):
        cs = O.Cosmo.from_vector(v)
        cs.transfer = transfer
        kw = {} if nonlinear == "takahashi2012" else {"nonlinear": nonlinear}
        return O.angular_cl(cs, ell, o, n_limber=n_limber, **kw)

    v = torch.tensor(row, dtype=torch.float64)
    return f(v), torch.autograd.functional.jacobian(f, v, strategy="forward-mode", vectorize=True)


def close(cl, jac, ref, tol):
    c, j = ref
    assert float(((cl.cpu() - c) / c).abs().max()) < tol
    err = (jac.cpu() - j).abs().amax(-2) / j.abs().amax(-2)  # per spectrum and parameter
    scale = j.abs().amax((0, 1)) / j.abs().amax((0, 1)).max()
    assert float((err * torch.clamp(scale, 0.01, 1.0)).max()) < tol, err.max()


@pytest.mark.parametrize("n_limber,n_ell,n_wl,n_nc", [
    (2, 1, 1, 0), (14, 1, 0, 1), (16, 33, 1, 1), (64, 65, 2, 1), (128, 7, 3, 2), (512, 31, 1, 0), (48, 9, 8, 8),
])
def test_sizes_vs_oracle(n_limber, n_ell, n_wl, n_nc):
    p, o = probes(n_wl, n_nc)
    ell = np.logspace(1, 3.5, n_ell) if n_ell > 1 else np.array([57.3])
    cl, jac = jc.autodiff.angular_cl_jacobian(batch([ROW]), ell, p, n_limber)
    close(cl[0], jac[0], oracle(ROW, ell, o, n_limber), 2e-12)


@pytest.mark.parametrize("nonlinear,transfer", [
    ("takahashi2012", "eisenhu"), ("smith2003", "eisenhu_osc"), ("smith2003", "eisenhu"), ("linear", "eisenhu_osc"),
    ("linear", "eisenhu"),
])
def test_operator_points_vs_oracle(nonlinear, transfer):
    p, o = probes(2, 1)
    ell = np.logspace(1, 3.5, 11)
    nl = jc.power.linear_matter_power if nonlinear == "linear" else functools.partial(jc.power.halofit, prescription=nonlinear)
    tf = functools.partial(jc.transfer.Eisenstein_Hu, type=transfer)
    cl, jac = jc.autodiff.angular_cl_jacobian(batch([ROW]), ell, p, 96, transfer_fn=tf, nonlinear_fn=nl)
    close(cl[0], jac[0], oracle(ROW, ell, o, 96, transfer, nonlinear), 2e-12)


@pytest.mark.parametrize("n_cosmo", [1, 40])
def test_one_cosmology_and_its_row_of_a_batch(n_cosmo):
    """Other splits of the a nodes: the sums differ by rounding only."""
    p, _ = probes(2, 1)
    ell = np.logspace(1, 3.5, 20)
    rows = np.array(ROW) * (1.0 + 0.02 * np.random.default_rng(2).standard_normal((n_cosmo, 8)))
    cl, jac = jc.autodiff.angular_cl_jacobian(batch(rows), ell, p, 256)
    one = jc.autodiff.angular_cl_jacobian(batch(rows[-1:]), ell, p, 256)
    fwd = jc.cl.angular_cl(batch(rows), ell, p, n_limber=256)
    assert float(((cl - fwd) / fwd).abs().max()) < 1e-13
    assert float(((cl[-1] - one[0][0]) / one[0][0]).abs().max()) < 1e-13
    assert float(((jac[-1] - one[1][0]).abs().amax((0, 1)) / one[1][0].abs().amax((0, 1))).max()) < 2e-13


def test_out_of_the_pairs_range():
    """ell of 10^7, a spectrum whose kernels do not overlap, a non-finite cosmology in a batch."""
    p, o = probes(1, 1)
    ell = np.array([30.0, 3e4, 2e7])
    cl, jac = jc.autodiff.angular_cl_jacobian(batch([ROW]), ell, p, 128)
    close(cl[0], jac[0], oracle(ROW, ell, o, 128), 1e-9)
    ell = np.array([30.0, 300.0])
    nz = [jc.redshift.smail_nz(1.0, 2.0, z, zmax=4.0) for z in (0.02, 1.0)]
    onz = [O.Smail(1.0, 2.0, z, 4.0, 1.0) for z in (0.02, 1.0)]
    pn = [jc.probes.NumberCounts(nz, jc.bias.constant_linear_bias(1.0))]
    cl, jac = jc.autodiff.angular_cl_jacobian(batch([ROW]), ell, pn, 128)
    close(cl[0], jac[0], oracle(ROW, ell, [O.Probe("nc", onz, bias=1.0)], 128), 1e-11)
    bad = np.array([ROW, ROW, ROW])
    bad[1, 2] = np.nan
    cl, jac = jc.autodiff.angular_cl_jacobian(batch(bad), ell, p, 128)
    ref = jc.autodiff.angular_cl_jacobian(batch([ROW, ROW, ROW]), ell, p, 128)
    assert torch.isnan(jac[1]).any()
    for i in (0, 2):
        assert torch.equal(jac[i], ref[1][i]) and torch.equal(cl[i], ref[0][i])
