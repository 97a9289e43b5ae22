"""The history scans' instances: one complex128 list of 1 to 20 vectors (blml_seg_dots2) against float64 sums on the host,
with an empty fit, fits around the tile of 64 and past one block; and the runner's two lists in one scan around 24 vectors
together, where the instance changes, with the memory filling and full (memory full of NaN against zeros, bit for bit)."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_history_mask import _fit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('np_', [1, 7, 8, 9, 16, 17, 20])
@pytest.mark.parametrize('B,K', [([0, 1, 63, 64, 65], [1, 1, 1, 1, 1]), ([5000, 17, 300], [4, 3, 2]), ([70001], [1])])
def test_one_list_of_complex128(cuda_device, np_, B, K):
    """Sums of n products of standard normals: 1e-15 n bounds their rounding in any order."""
    from blml_b200 import _lib
    from blml_b200._lib import call, ptrs
    from blml_b200.sweep import _Seg
    rng = np.random.default_rng(np_)
    F = len(B); n_f = np.array(B) * np.array(K)
    off = np.concatenate([[0], np.cumsum(n_f)]); boff = np.concatenate([[0], np.cumsum(B)])
    segs = (_Seg * F)(*[_Seg(int(off[f]), int(boff[f]), int(B[f]), int(K[f]), 0) for f in range(F)])
    st_t = torch.frombuffer(bytearray(segs), dtype=torch.uint8).cuda()
    n = int(off[-1])
    v = [rng.standard_normal(n) + 1j * rng.standard_normal(n) for _ in range(np_ + 3)]
    d = [torch.from_numpy(a).cuda() for a in v]
    st = torch.cuda.current_stream().cuda_stream
    for with_x in (True, False):
        part = torch.full((48 * 16384,), np.nan, dtype=torch.float64, device='cuda')
        out = torch.full((F * (2 * np_ + 3),), np.nan, dtype=torch.float64, device='cuda')
        call('blml_seg_dots2', _lib.F64, F, st_t.data_ptr(), 1, np_, ptrs(d[:np_]), d[np_].data_ptr(), d[np_ + 1].data_ptr(),
             d[np_ + 2].data_ptr() if with_x else C.c_void_p(0), part.data_ptr(), out.data_ptr(), st)
        got = out.cpu().numpy().reshape(F, -1)
        for f in range(F):
            s = slice(int(off[f]), int(off[f + 1]))
            b0, b1, x = v[np_][s], v[np_ + 1][s], v[np_ + 2][s]
            dot = lambda p, q: float(np.sum(p.real * q.real + p.imag * q.imag))
            want = [dot(a[s], b0) for a in v[:np_]] + [dot(a[s], b1) for a in v[:np_]] + \
                [dot(b0, b0), dot(b1, b1), dot(x, x) if with_x else 0.0]
            assert np.all(np.abs(got[f] - want) <= 1e-15 * max(int(n_f[f]), 1))


@pytest.mark.parametrize('h32', [False, True])
@pytest.mark.parametrize('m,iters', [(12, 7), (12, 30), (13, 8), (13, 30), (20, 30)])
def test_two_lists(cuda_device, m, iters, h32):
    l0, e0 = _fit(0.0, m, iters, np.float64, h32, 2)
    l1, e1 = _fit(float('nan'), m, iters, np.float64, h32, 2)
    assert np.all(np.isfinite(l1)) and np.all(np.isfinite(e1))
    np.testing.assert_array_equal(l0, l1)
    np.testing.assert_array_equal(e0, e1)
