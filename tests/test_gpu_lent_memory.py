"""Groups and batch runners in memory lent by torch's allocator: on another stream than the default one, launched on a
second stream, after the memory was just given back by other work; and a lender that has none left."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch():
    from blml_b200 import workloads
    rng = np.random.default_rng(0)
    shapes = [(64, 64), (48, 64), (51, 50)]
    modes = [workloads.pball_modes(s, 0.3) for s in shapes]
    return [rng.poisson(3.0, s).astype(float) for s in shapes], modes


def test_fit_on_a_side_stream_equals_default_stream(cuda_device):
    from blml_b200.sweep import BLMLBinnedBatch
    counts, modes = _batch()
    a = BLMLBinnedBatch(tol=1e-9, max_sweeps=6).fit(counts, modes)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        dirt = torch.full((1 << 24,), float('nan'), device='cuda', dtype=torch.float64)
        dirt.mul_(2.0)
        del dirt                                              # the fit's memory: still being written on this stream
        batch = BLMLBinnedBatch(tol=1e-9, max_sweeps=6)
        b = batch.fit(counts, modes)
        cert = batch.certificate()
    assert np.all(np.isfinite(cert))
    for x, y in zip(a, b):
        assert x.loglik_ == y.loglik_ and x.n_sweeps_ == y.n_sweeps_
        np.testing.assert_array_equal(x.density_, y.density_)


def test_group_on_a_second_stream(cuda_device):
    from blml_b200 import _lib
    from blml_b200.sweep import BLMLBinnedBatch, _Group
    _, modes = _batch()
    from blml_b200.spec import parse_modes
    sp, _ = parse_modes(modes[0], 2)
    p, _ = BLMLBinnedBatch()._plan(sp[0], (64, 64), _lib.F64)
    x = torch.randn(3, 64, 64, dtype=torch.complex128, device='cuda')
    y = torch.empty_like(x); ref = torch.empty_like(x)
    st = torch.cuda.current_stream().cuda_stream
    p.apply(x, ref, 3, True, st)
    off = [i * 4096 for i in range(3)]
    g = _Group([p] * 3, x, off, y, off, True)
    other = torch.cuda.Stream()
    other.wait_stream(torch.cuda.current_stream())
    g(other.cuda_stream)
    del g
    junk = [torch.full((1 << 20,), float('nan'), device='cuda') for _ in range(4)]      # may not take the group's memory early
    torch.cuda.synchronize()
    assert len(junk) == 4
    torch.testing.assert_close(y, ref, rtol=1e-13, atol=0)


def test_lender_without_memory(cuda_device):
    from blml_b200 import _lib, workloads
    from blml_b200.sweep import BLMLBinnedBatch
    from blml_b200.spec import parse_modes
    sp, _ = parse_modes(workloads.pball_modes((64, 64), 0.3), 2)
    p, _ = BLMLBinnedBatch()._plan(sp[0], (64, 64), _lib.F64)
    x = torch.zeros(64, 64, dtype=torch.complex128, device='cuda')
    fn = _lib.ALLOC_FN(lambda n, ctx: None)
    h = C.c_void_p()
    arr = (C.c_void_p * 1)(p._h.value)
    one = np.ones(1, np.int32); off = np.zeros(1, np.int64)
    with pytest.raises(_lib.BLMLError, match='allocation'):
        _lib.call('blml_group_create_with', 1, C.cast(arr, C.c_void_p), _lib.host_ptr(one), 1, x.data_ptr(),
                  _lib.host_ptr(off), x.data_ptr(), _lib.host_ptr(off), fn, None, None, C.byref(h))
    assert not h.value
