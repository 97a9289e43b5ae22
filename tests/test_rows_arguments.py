"""Row sums refuse missing tables and negative counts with an argument error, before anything is divided or launched (no GPU
needed: nothing else is looked at)."""
import ctypes as C

import pytest

from blml_b200 import _lib

ARG = -1         # BLML_ERR_ARG


def _masks():
    return (C.c_uint32 * 1)(1)


@pytest.mark.parametrize('R,M', [(-1, 5), (-127, 5), (-128, 5), (-254, 5), (-300, 5), (-1, 0), (5, -1), (0, -1), (-1, -1)])
def test_negative_counts(R, M):
    tb = _lib.Tables()
    L = _lib.lib()
    assert L.blml_rows(C.byref(tb), None, R, None, M, None, 0, None, None, None) == ARG
    assert b'negative' in L.blml_last_error()
    assert L.blml_rows_ws(C.byref(tb), None, R, None, M, None, 0, None, None, None, 0, None) == ARG
    assert b'negative' in L.blml_last_error()
    assert L.blml_rows_multi(C.byref(tb), None, R, None, M, None, 1, _masks(), None, None) == ARG
    assert b'negative' in L.blml_last_error()
    assert L.blml_rows_workspace(R, M, 0) == 0


def test_no_tables():
    L = _lib.lib()
    for R, M in ((5, 5), (0, 5), (5, 0)):
        assert L.blml_rows(None, None, R, None, M, None, 0, None, None, None) == ARG
        assert L.blml_rows_ws(None, None, R, None, M, None, 0, None, None, None, 0, None) == ARG


@pytest.mark.gpu
def test_plan_workspace_without_rows(cuda_device):
    import numpy as np
    import torch
    from blml_b200.local_gpu import ProductKernel, _struct, dev_tab, rank_coords
    Z = np.arange(12, dtype=np.int64).reshape(-1, 1)
    tab = ProductKernel(['sinc'], [None]).tables(np.array([0.3]), [None], np.ones(1), Z)
    Zd = torch.as_tensor(rank_coords(Z, tab)).cuda()
    h = C.c_void_p()
    t = dev_tab(tab, Zd.device)
    _lib.call('blml_rows_plan_create', _struct(tab, t, False, False), Zd.data_ptr(), 12, None, C.byref(h))
    assert _lib.lib().blml_rows_plan_workspace(h, 0, 12) == 0 and _lib.lib().blml_rows_plan_workspace(h, 3, 12) > 0
    _lib.lib().blml_rows_plan_destroy(h)
