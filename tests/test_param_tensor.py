"""Cosmology.param_tensor with host values (one upload), tensors and both mixed."""
import numpy as np
import pytest
import torch

import jax_cosmo_gb300 as jc

NAMES = ["Omega_c", "Omega_b", "h", "n_s", "sigma8", "Omega_k", "w0", "wa"]
ROW = [0.25, 0.05, 0.7, 0.96, 0.8, 0.0, -1.0, 0.0]


@pytest.mark.parametrize("kinds", ["n" * 8, "a" * 8, "nanananan"[:8], "tttttttt", "ntntntnt", "natnatna"])
@pytest.mark.parametrize("B", [None, 1, 3])
def test_values_and_gradients(kinds, B):
    vals, want = {}, np.tile(ROW, ((B or 1) if kinds != "n" * 8 else 1, 1))  # numbers alone are no batch
    for i, (n, k) in enumerate(zip(NAMES, kinds)):
        if k == "n" or B is None and k == "a":
            vals[n] = ROW[i] if i % 2 else np.float64(ROW[i])
        elif k == "a":
            vals[n] = ROW[i] + 0.01 * np.arange(B)
            want[:, i] = vals[n]
        else:
            vals[n] = torch.tensor(ROW[i] if B is None else [ROW[i]] * B, dtype=torch.float64, requires_grad=True)
    c = jc.Cosmology(**vals)
    p = c.param_tensor("cpu", differentiable=True)
    assert p.shape == want.shape and p.dtype == torch.float64 and p.is_contiguous()
    assert np.array_equal(p.detach().numpy(), want)
    assert p.requires_grad == ("t" in kinds)
    if p.requires_grad:
        p.sum().backward()
        for n, k in zip(NAMES, kinds):
            if k == "t":
                assert torch.equal(vals[n].grad, torch.ones_like(vals[n]))
    assert not c.param_tensor("cpu").requires_grad


def test_refused():
    with pytest.raises(ValueError):
        jc.Cosmology(**{**dict(zip(NAMES, ROW)), "h": np.array([0.6, 0.7]), "n_s": np.ones(3)}).param_tensor("cpu")
    with pytest.raises(ValueError):
        jc.Cosmology(**{**dict(zip(NAMES, ROW)), "h": float("inf")}).param_tensor("cpu")
    with pytest.raises(RuntimeError):
        jc.Cosmology(**{**dict(zip(NAMES, ROW)), "h": np.ones((2, 2))}).param_tensor("cpu")
