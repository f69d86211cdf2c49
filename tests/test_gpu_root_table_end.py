"""Cosmologies whose non-linear scale lies past the end of the sigma^2(R) table (R above
10 Mpc/h: sigma_8 of 2 and more, or little matter): the root is taken on the table's
last segment there, in C_ell, its Jacobian and the vector-Jacobian product alike.

Tolerances: float64 as for ordinary cosmologies, 1e-11 of the oracle (C_ell) and of
a column's largest entry (Jacobian); fp32c 1e-4 of each."""
import functools

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import jax_cosmo_gb300 as jc  # noqa: E402
from oracle import jc_oracle as O  # noqa: E402

ROWS = {
    "sigma8 2": [0.27, 0.047, 0.69, 0.96, 2.0, 0.01, -0.95, 0.1],
    "sigma8 3": [0.16, 0.037, 0.87, 0.97, 3.0, -0.02, -0.76, 0.0],
    "little matter": [0.01, 0.037, 0.87, 0.97, 0.9, -0.02, -0.76, 0.0],
}
ELL = np.geomspace(10, 1000, 5)


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def cosmo(row, n=1):
    t = torch.tensor([row] * n, dtype=torch.float64, device="cuda")
    return jc.Cosmology(*[t[:, i] for i in range(8)])


@pytest.mark.parametrize("row", list(ROWS))
@pytest.mark.parametrize("transfer,nonlinear", [("eisenhu", "takahashi2012"), ("eisenhu_osc", "takahashi2012"),
                                                ("eisenhu_osc", "smith2003")])
def test_past_the_end(row, transfer, nonlinear):
    row = ROWS[row]
    probes = [jc.probes.WeakLensing([jc.redshift.smail_nz(1.0, 2.0, 1.2, zmax=4.0)])]
    opt = dict(n_limber=128, transfer_fn=functools.partial(jc.transfer.Eisenstein_Hu, type=transfer),
               nonlinear_fn=functools.partial(jc.power.halofit, prescription=nonlinear))

    def f(v):
        cs = O.Cosmo.from_vector(v)
        cs.transfer = transfer
        return O.angular_cl(cs, ELL, [O.Probe("wl", [O.Smail(1.0, 2.0, 1.2, 4.0, 1.0)])], n_limber=128, nonlinear=nonlinear)

    v = torch.tensor(row, dtype=torch.float64)
    cl, jac = f(v), torch.autograd.functional.jacobian(f, v, strategy="forward-mode", vectorize=True)
    scale = jac.abs().amax(1)
    for n in (1, 130):  # both forms of the batch
        got = jc.cl.angular_cl(cosmo(row, n), ELL, probes, **opt)
        c, j = jc.autodiff.angular_cl_jacobian(cosmo(row, n), ELL, probes, **opt)
        for x in (got[-1], c[-1]):
            assert float(((x.cpu() - cl) / cl).abs().max()) < 1e-11
        assert float(((j[-1].cpu() - jac).abs().amax(1) / scale).max()) < 1e-11
        f32 = jc.cl.angular_cl(cosmo(row, n), ELL, probes, precision="fp32c", **opt)
        c, j = jc.autodiff.angular_cl_jacobian(cosmo(row, n), ELL, probes, precision="fp32c", **opt)
        for x in (f32[-1], c[-1]):
            assert float(((x.cpu() - cl) / cl).abs().max()) < 1e-4
        assert float(((j[-1].cpu() - jac).abs().amax(1) / scale).max()) < 1e-4
