"""A kernel's dynamic shared-memory limit belongs to the process: every launch goes
through the one function that only raises it (under its lock), and threads with
surveys of different sizes run side by side."""
import glob
import os
import re
import threading

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jax_cosmo_gb300", "csrc")


def test_the_limit_is_set_in_one_place():
    found = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        with open(path) as f:
            found += [os.path.basename(path)] * len(re.findall("cudaFuncAttributeMaxDynamicSharedMemorySize", f.read()))
    assert found == ["jcg_api.cu"], found


@pytest.mark.gpu
def test_threads_with_surveys_of_different_sizes():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    import jax_cosmo_gb300 as jc

    def job(n_wl, n_ell, n):
        nz = [jc.redshift.smail_nz(1.0, 2.0, 0.4 + 0.1 * i, gals_per_arcmin2=10.0, zmax=4.0) for i in range(n_wl)]
        p, ell = [jc.probes.WeakLensing(nz, sigma_e=0.26)], np.logspace(1, 3, n_ell)
        c = jc.Planck15()
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(n):
                cl, jac = jc.autodiff.angular_cl_jacobian(c, ell, p, 64)
                f32 = jc.cl.angular_cl(c, ell, p, precision="fp32c", n_limber=64)
                cov = jc.cl.gaussian_cl_covariance(ell, p, cl, jc.cl.noise_cl(ell, p), sparse=True)
                ll = jc.likelihood.gaussian_log_likelihood(cl.flatten() * 0.9, cl.flatten(), cov)
            torch.cuda.current_stream().synchronize()
            return [t.cpu() for t in (cl, jac, f32, ll)]

    sizes = [(1, 9), (7, 40), (3, 23), (5, 64)]
    want, got, errors = [job(*s, 1) for s in sizes], [None] * len(sizes), []

    def run(i):
        try:
            got[i] = job(*sizes[i], 150)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(sizes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for w, g in zip(want, got):
        for name, a, b in zip(("cl", "jac", "fp32c", "loglike"), w, g):
            assert bool(torch.isfinite(a).all()) and torch.equal(a, b), name
