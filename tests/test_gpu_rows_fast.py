"""The rows kernel for tables without groups (csrc/pairs.cu, k_rows_fast) against the same sums taken from the table
arrays on the CPU in float64: 1 to 8 columns of every kind it unfolds (offset, circular, rank), values and derivative
entries, rows and columns around the block and chunk sizes, sorted and unsorted bins, large coordinates."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(kinds, R, M, seed, want=(), shift=0):
    from blml_b200.local_gpu import ProductKernel
    rng = np.random.default_rng(seed)
    d = len(kinds)
    Z = np.zeros((R + M, d), np.int64)
    for k, kd in enumerate(kinds):
        if kd == 'dirichlet':
            Z[:, k] = rng.integers(0, 24, R + M)
        elif kd == 'rank':                       # few values far apart: a rank table
            Z[:, k] = shift + 1000 * rng.integers(0, 5, R + M)
        else:
            Z[:, k] = shift + rng.integers(0, 40, R + M)
    names = ['sinc' if kd == 'rank' else kd for kd in kinds]
    per = [24.0 if kd == 'dirichlet' else None for kd in kinds]
    fc = np.array([0.3 / (1000 if kd == 'rank' else 1) for kd in kinds]) * (1 + 0.1 * np.arange(d))
    tab = ProductKernel(names, per).tables(fc, per, np.ones(d), Z, want=list(want))
    return Z[:R], Z[R:], rng.standard_normal(M), tab


def _reference(A, B, w, tab, grad):
    from blml_b200.local_gpu import rank_coords
    A, B = rank_coords(A, tab), rank_coords(B, tab)
    d = A.shape[1]
    fac, raw = [], []
    for k in range(d):
        a, b = A[:, k][:, None], B[:, k][None, :]
        code = int(tab['kinds'][k])
        if code == 3:
            i = a * tab['mk'][k] + b
        elif code == 0:
            i = a - b + tab['Jk'][k]
        else:
            i = np.abs(a - b); i = np.minimum(i, tab['nbins'][k] - i)
        raw.append(a * tab['mk'][k] + b if code == 3 else a - b + tab['Jk'][k])
        fac.append(tab['T'][tab['base'][k] + i])
    s = np.prod(fac, 0) @ w
    ds = []
    for q in range(int(tab['nW']) if grad else 0):
        k = int(tab['wcol'][q])
        f = [tab['dT'][tab['dbase'][q] + raw[k]] if j == k else fac[j] for j in range(d)]
        ds.append(np.prod(f, 0) @ w)
    scale = np.abs(np.prod(fac, 0)) @ np.abs(w)
    return s, (np.stack(ds, 1) if ds else None), scale


O, C, K = 'sinc', 'dirichlet', 'rank'


@pytest.mark.parametrize('f32', [False, True])
@pytest.mark.parametrize('kinds,R,M,srt', [((O,), 1, 1, True), ((C,), 127, 255, False), ((K,), 129, 257, True),
                                           ((O, C), 256, 256, True), ((K, O), 257, 511, False),
                                           ((O, O, C), 1000, 1025, True), ((C, K, O, O), 300, 700, False),
                                           ((O,) * 5, 600, 3000, True), ((O, C, K, O, C, O), 130, 300, True),
                                           ((O,) * 7, 50, 260, False), ((O, O, C, O, K, O, O, C), 140, 513, True),
                                           ((O, O, O), 80000, 300, True)])
def test_rows_values(cuda_device, kinds, R, M, srt, f32):
    """Float64 tables: rounding of d products and a sum (1e-13 of sum |terms|). Float32 tables: every factor and product
    rounded to 24 bits, 2 d 2^-24 of sum |terms|."""
    from blml_b200.local_gpu import rows
    A, B, w, tab = _case(kinds, R, M, seed=R + M, shift=3_000_000_000 if kinds[0] == O else 0)
    if srt:
        B = B[np.lexsort(B.T[::-1])]
    s, _ = rows(A, B, w, tab, f32=f32)
    sel = np.linspace(0, R - 1, min(R, 400)).astype(int)
    ref, _, scale = _reference(A[sel], B, w, tab, False)
    tol = 2 * len(kinds) * 2.0 ** -24 if f32 else 1e-13
    assert np.all(np.abs(s[sel] - ref) <= tol * scale)


@pytest.mark.parametrize('f32', [False, True])
@pytest.mark.parametrize('kinds,want', [((O,), [(0, 'fc')]), ((O, C), [(0, 'fc'), (0, 'shift')]),
                                        ((K, O, C), [(1, 'shift'), (0, 'fc'), (1, 'fc')]),
                                        ((O, O, O, O, O), [(4, 'fc'), (0, 'shift'), (2, 'fc'), (2, 'shift'), (1, 'fc')]),
                                        ((C, O, K, O, O, C, O, O), [(k, p) for k in (1, 2, 7, 4) for p in ('fc', 'shift')])])
def test_rows_derivatives(cuda_device, kinds, want, f32):
    from blml_b200.local_gpu import rows
    A, B, w, tab = _case(kinds, 259, 520, seed=len(kinds), want=want)
    s, ds = rows(A, B, w, tab, grad=True, f32=f32)
    ref, dref, scale = _reference(A, B, w, tab, True)
    tol = 2 * len(kinds) * 2.0 ** -24 if f32 else 1e-13
    top = max(1.0, np.abs(tab['dT']).max() / min(np.abs(tab['T']).max(), 1.0))
    assert np.all(np.abs(s - ref) <= tol * scale)
    assert np.all(np.abs(ds - dref) <= tol * top * max(scale.max(), np.abs(w).sum() * np.abs(tab['T']).max() ** (len(kinds) - 1)))


def test_rows_workspace_checked(cuda_device):
    from blml_b200 import _lib
    from blml_b200.local_gpu import dev_tab, _struct
    A, B, w, tab = _case((O, C), 10, 20, seed=0)
    t = dev_tab(tab, 'cuda')
    dev = lambda a: torch.as_tensor(a).cuda()  # noqa: E731
    A, B, w, s = dev(A), dev(B), dev(w), torch.empty(10, dtype=torch.float64, device='cuda')
    need = int(_lib.lib().blml_rows_workspace(10, 20, 0))
    ws = torch.empty(need, dtype=torch.uint8, device='cuda')
    args = (_struct(tab, t, False, False), A.data_ptr(), 10, B.data_ptr(), 20, w.data_ptr(), 0, s.data_ptr(), None)
    st = torch.cuda.current_stream().cuda_stream
    with pytest.raises(_lib.BLMLError):
        _lib.call('blml_rows_ws', *args, ws.data_ptr(), need - 1, st)
    _lib.call('blml_rows_ws', *args, ws.data_ptr(), need, st)
    out = torch.empty_like(s)
    _lib.call('blml_rows', *args[:7], out.data_ptr(), None, st)
    assert torch.equal(s, out)
