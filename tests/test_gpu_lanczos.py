"""blml_lanczos_step (csrc/lanczos.cu) against NumPy: bases around the kernels' groups of 8, 16 and 64 vectors, lattices
smaller and larger than a block's chunk and odd ones, first and later steps, launches over some of the fits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(64, 64), (5, 7), (51, 50)]


@pytest.mark.parametrize('rows', [[0, 1, 2], [2, 0]])
@pytest.mark.parametrize('chunk', [512, 768])
@pytest.mark.parametrize('j', [0, 1, 6, 7, 8, 15, 16, 47, 48, 63, 64, 130])
def test_step(cuda_device, j, chunk, rows):
    """Every value is a sum of at most 4,096 products of unit vectors: 1e-13 of the largest."""
    from blml_b200 import _lib, workloads
    from blml_b200._lib import call
    from blml_b200.spec import parse_modes
    from blml_b200.sweep import BLMLBinnedBatch, _Group, _Seg
    dev = torch.device('cuda')
    plans = []
    for s in SHAPES:
        sp, _ = parse_modes(workloads.pball_modes(s, 0.3), 2)
        plans.append(BLMLBinnedBatch()._plan(sp[0], s, _lib.F64)[0])
    B = np.array([a * b for a, b in SHAPES]); off = np.concatenate([[0], np.cumsum(B)]); n = int(off[-1])
    rng = np.random.default_rng(j)
    V = np.zeros((j + 1, n))
    for f in range(3):
        k = min(j + 1, int(B[f]) - 1)
        V[:k, off[f]:off[f + 1]] = np.linalg.qr(rng.standard_normal((int(B[f]), k)))[0].T
    w0 = rng.standard_normal(n); scale0 = rng.uniform(0.5, 2.0, 3); dh = rng.uniform(0.5, 1.5, n)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a)).to(dev)
    Vt, wt, st_, dt = t(V), t(w0), t(scale0), t(dh)
    tmp, sv = torch.zeros(n, dtype=torch.float64, device=dev), torch.zeros(n, dtype=torch.float64, device=dev)
    segs = (_Seg * len(rows))(*[_Seg(int(off[f]), int(off[f]), int(B[f]), 1, 0) for f in rows])
    segs_t = torch.frombuffer(bytearray(segs), dtype=torch.uint8).to(dev)
    tab = [(r, c) for r, f in enumerate(rows) for c in range(-(-int(B[f]) // chunk))]
    tab_t = t(np.array(tab, np.int32)); fid = t(np.array(rows, np.int32)); cnt = t(np.zeros(len(rows), np.int32))
    grp = _Group([plans[f] for f in rows], tmp, off[rows], sv, off[rows], False)
    part = torch.empty(64 * len(tab), dtype=torch.float64, device=dev); coef = torch.empty(64 * 3, dtype=torch.float64, device=dev)
    al = torch.full((3,), 7.0, dtype=torch.float64, device=dev); be = al.clone()
    st = torch.cuda.current_stream().cuda_stream
    call('blml_lanczos_step', len(rows), segs_t.data_ptr(), fid.data_ptr(), len(tab), tab_t.data_ptr(), chunk, grp.on(st),
         Vt.data_ptr(), n, j, dt.data_ptr(), tmp.data_ptr(), sv.data_ptr(), wt.data_ptr(), part.data_ptr(), cnt.data_ptr(),
         coef.data_ptr(), al.data_ptr(), be.data_ptr(), st_.data_ptr(), st)
    assert not cnt.any()
    for f in range(3):
        sl = slice(off[f], off[f + 1])
        if f not in rows:
            assert al[f] == 7.0 and be[f] == 7.0
            np.testing.assert_array_equal(wt[sl].cpu().numpy(), w0[sl])
            continue
        Vf = V[:, sl].copy()
        if j:
            Vf[j] = scale0[f] * w0[sl]
        np.testing.assert_array_equal(Vt[j, sl].cpu().numpy(), Vf[j])
        x = torch.as_tensor(dh[sl] * Vf[j]).reshape((1,) + SHAPES[f]).to(dev)
        y = torch.empty_like(x)
        plans[f].apply(x, y, 1, False, st)
        w = dh[sl] * y.cpu().numpy().ravel()
        big = np.abs(w).max()
        first = None
        for ps in range(2):
            for q0 in range(0, j + 1, 64):
                q1 = min(j + 1, q0 + 64)
                c = Vf[q0:q1] @ w
                if ps == 0 and q1 == j + 1:
                    first = c[j - q0]
                w = w - Vf[q0:q1].T @ c
        tol = 1e-13 * max(1.0, big) * max(1.0, np.abs(Vf[j]).max() ** 2 * B[f]) * 10
        assert abs(al[f].item() - first) <= tol * np.sqrt(B[f])
        assert np.abs(wt[sl].cpu().numpy() - w).max() <= tol * np.sqrt(B[f])
        b = np.linalg.norm(w)
        assert abs(be[f].item() - b) <= tol * B[f]
        got = be[f].item()
        assert st_[f].item() == (1.0 / got if got > 0 else 0.0)


def test_launches_over_any_number_of_fits(cuda_device):
    """A batch whose open fits shrink through odd and even numbers: the certificates equal each fit's own."""
    from blml_b200 import workloads
    from blml_b200.sweep import BLMLBinnedBatch
    rng = np.random.default_rng(1)
    shapes = [(16 + 8 * (i % 4), 24 + 4 * (i % 3)) for i in range(9)]
    counts = [rng.poisson(0.5 + i, s).astype(float) + 1.0 for i, s in enumerate(shapes)]
    modes = [workloads.pball_modes(s, 0.05 + 0.04 * i) for i, s in enumerate(shapes)]
    b = BLMLBinnedBatch(tol=1e-9, max_sweeps=2)
    b.fit(counts, modes)
    both = b.certificate()
    assert np.all(np.isfinite(both))
    for i in (0, 4, 8):
        one = BLMLBinnedBatch(tol=1e-9, max_sweeps=2)
        one.fit(counts[i:i + 1], modes[i:i + 1])
        assert abs(one.certificate()[0] - both[i]) <= 1e-5 * abs(both[i])


@pytest.mark.parametrize('n', [1, 2, 3, 6, 33, 64, 130, 1500])
def test_check(cuda_device, n):
    """The two top eigenvalues within 4 n eps of the largest in size, the last component (exact up to the eigenvalue's
    error over the gap) within 1e-7, for random, graded, split, repeated and zero matrices, of some of the fits."""
    from blml_b200 import _lib
    rng = np.random.default_rng(n)
    F = 7
    a, b = rng.standard_normal((n, F)), np.abs(rng.standard_normal((n, F))) + 0.1
    a[:, 1] *= 1e-150; b[:, 1] *= 1e-150
    a[:, 2] = 1e5 * 0.5 ** np.arange(n); b[:, 2] = 1e3 * 0.5 ** np.arange(n)
    b[n // 2, 3] = 0.0                                        # two blocks
    a[:, 4] = 2.0; b[:, 4] = 1e-9                             # a cluster
    a[:, 5] = 0.0; b[:, 5] = 0.0
    a[:, 6] = np.abs(a[:, 6]) + 1e6                           # close to a multiple of the identity
    ab = torch.as_tensor(np.stack([a, b], 1)).cuda()
    rows = np.array([6, 0, 1, 2, 3, 4, 5], np.int32)[:7 if n % 2 else 6]
    fid = torch.as_tensor(rows).cuda()
    out = torch.full((F, 4), 9.0, dtype=torch.float64, device='cuda')
    work = torch.empty(4 * n * F, dtype=torch.float64, device='cuda')
    _lib.call('blml_lanczos_check', len(rows), fid.data_ptr(), F, ab.data_ptr(), n - 1, work.data_ptr(), out.data_ptr(),
              torch.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy()
    for f in range(F):
        if f not in rows:
            assert np.all(got[f] == 9.0)
            continue
        T = np.diag(a[:, f]) + np.diag(b[:-1, f], 1) + np.diag(b[:-1, f], -1)
        ev, vec = np.linalg.eigh(T)
        big = np.abs(ev).max()
        assert abs(got[f, 0] - ev[-1]) <= 4 * n * 2.3e-16 * big + 1e-300
        if n > 1:
            assert abs(got[f, 1] - ev[-2]) <= 4 * n * 2.3e-16 * big + 1e-300
        else:
            assert np.isnan(got[f, 1]) or f == 5
        assert got[f, 3] == b[n - 1, f]
        gap = (ev[-1] - ev[-2]) / big if n > 1 and big > 0 else 1.0
        if f not in (4, 5) and gap > 1e-6:
            assert abs(got[f, 2] - abs(vec[-1, -1])) <= 1e-7
