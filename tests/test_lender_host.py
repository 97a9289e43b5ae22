"""Memory lent to the library goes back when its lender is dropped, without Python's cyclic collector."""
import gc
import weakref

import torch

from blml_b200 import _lib


def test_lent_memory_dies_with_its_lender():
    on = gc.isenabled()
    gc.disable()
    try:
        lender = _lib.Lender(torch.device('cpu'))
        at = [lender.fn(n, None) for n in (1 << 20, 16)]
        assert [t.data_ptr() for t in lender.tensors] == at and [t.numel() for t in lender.tensors] == [1 << 20, 16]
        dead = [weakref.ref(t) for t in lender.tensors]
        del lender
        assert [r() for r in dead] == [None, None]
    finally:
        if on:
            gc.enable()


def test_lender_without_memory_returns_null():
    lender = _lib.Lender(torch.device('cpu'))
    assert lender.fn(1 << 62, None) is None and lender.tensors == []
