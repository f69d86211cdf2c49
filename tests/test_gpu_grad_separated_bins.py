"""The float64 Jacobian of narrow bins far apart (kernels that overlap below 2^-66 of
their largest values): such a cosmology is computed by the float64 kernels, and the
integral in float pairs is not computed for it before."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

import jax_cosmo_gb300 as jc  # noqa: E402
from oracle import jc_oracle as O  # noqa: E402

ROW = [0.27, 0.047, 0.69, 0.96, 0.81, 0.01, -0.95, 0.1]
ELL = np.logspace(1, 3, 40)


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")


def probes(a, b):
    nz = [jc.redshift.smail_nz(a, b, z, zmax=4.0) for z in (0.4, 0.8, 1.2)]
    onz = [O.Smail(a, b, z, 4.0, 1.0) for z in (0.4, 0.8, 1.2)]
    return [jc.probes.NumberCounts(nz, jc.bias.constant_linear_bias(1.2))], [O.Probe("nc", onz, bias=1.2)]


def batch(n):
    r = np.array([ROW] * n)
    r[:, 0] += 0.001 * np.arange(n)
    return jc.Cosmology(*[torch.tensor(r[:, i], dtype=torch.float64, device="cuda") for i in range(8)])


def test_values_in_a_batch():
    """Tolerance: as of the float64 kernels' own tests, 1e-11 of a spectrum's largest entry."""
    p, o = probes(300.0, 120.0)
    cl, jac = jc.autodiff.angular_cl_jacobian(batch(3), ELL[::8], p, 128)

    def f(v):
        return O.angular_cl(O.Cosmo.from_vector(v), ELL[::8], o, n_limber=128)

    for b in (0, 2):
        v = torch.tensor(ROW, dtype=torch.float64)
        v[0] += 0.001 * b
        ref = torch.autograd.functional.jacobian(f, v, strategy="forward-mode", vectorize=True)
        assert float(((cl[b].cpu() - f(v)) / f(v)).abs().max()) < 1e-11
        big = ref.abs().amax(1)
        err = (jac[b].cpu() - ref).abs().amax(1) / big
        scale = big / big.amax(1, keepdim=True)
        assert float((err * torch.clamp(scale, 0.01, 1.0)).max()) < 1e-11


def pairs_time(p):
    """Device time of the integral in float pairs of one call of 16 cosmologies."""
    from torch.profiler import ProfilerActivity, profile

    c = batch(16)
    jc.autodiff.angular_cl_jacobian(c, ELL, p, 256)
    torch.cuda.synchronize()
    for _ in range(2):  # the profiler's first session sets itself up
        with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as prof:
            jc.autodiff.angular_cl_jacobian(c, ELL, p, 256)
            torch.cuda.synchronize()
    t = [e.device_time for e in prof.events() if "grad_limber64_kernel" in e.name]
    if not t:
        pytest.skip("no kernel times from the profiler")
    return sum(t)


def test_the_integral_in_pairs_is_left_out():
    both, apart = pairs_time(probes(1.0, 2.0)[0]), pairs_time(probes(300.0, 120.0)[0])
    assert apart < 0.3 * both, (apart, both)
