"""A tensor lives as long as the pointer that is passed on for it."""
import gc
import weakref

import torch

from jax_cosmo_gb300 import _lib


def test_pointer_holds_its_tensor():
    t = torch.arange(6.0).expand(2, 6).contiguous()
    alive, address = weakref.ref(t), t.data_ptr()
    p = _lib.ptr(t)
    del t
    gc.collect()
    assert p.value == address and alive() is not None
    del p
    gc.collect()
    assert alive() is None
    assert _lib.ptr(None) is None


def test_temporaries_live_through_the_call(monkeypatch):
    alive = []

    class Library:
        def __getattr__(self, name):
            def f(*args):
                alive.extend(w() is not None for w in tensors)
                return 0
            return f

    tensors = []
    data_ptr = torch.Tensor.data_ptr

    def spy(t):
        tensors.append(weakref.ref(t))
        return data_ptr(t)

    monkeypatch.setattr(torch.Tensor, "data_ptr", spy)
    monkeypatch.setattr(_lib, "load", lambda: Library())
    go = torch.tensor(2.0).expand(3)
    _lib.call("anything", _lib.ptr(go.contiguous()), _lib.ptr(torch.zeros(4)))
    assert alive == [True, True]
