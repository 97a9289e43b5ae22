"""The points path of BLMLQuick on the GPU against the reference's own point fits (tests/golden/points.npz): the same
bins in the same order, the coefficients of the convex real rank-1 fit (both solved to max|rho| < 1e-8) within 1e-6 of
their largest, predict / sqrt_density at off-lattice query points within 1e-6 of the largest value; the point kernel
alone (blml_point_rows at the reference's coefficients) to 1e-11; float32 fits within 1e-3."""
import numpy as np
import pytest
import torch

from conftest import golden
from golden_cases import POINT_SPECS

pytestmark = pytest.mark.gpu


def _fit(name, dtype=np.float64):
    from blml_b200.quick import BLMLQuick
    g = golden('points.npz')[name]
    modes, n, weighted, seed = POINT_SPECS[name]
    m = BLMLQuick(dtype=dtype, tol=1e-8).fit(g['X'], modes, sample_weight=g['sw'] if weighted else None)
    return g, m


def _rel(a, b):
    return float(np.max(np.abs(np.ravel(a) - np.ravel(b))) / np.max(np.abs(b)))


@pytest.mark.parametrize('name', list(POINT_SPECS))
def test_point_fit_matches_reference(cuda_device, name):
    g, m = _fit(name)
    assert np.array_equal(m.Z_, g['Z']) and np.array_equal(m.w_pts_, g['w']) and np.array_equal(m._h_vec, g['h'])
    assert m.n_samples_ == float(g['n'])
    assert _rel(m.e_hat_, g['e_hat']) <= 1e-6
    assert _rel(m.predict(g['Xq']), g['predict']) <= 1e-6
    assert _rel(m.sqrt_density(g['Xq']), g['sqrt_density']) <= 1e-6


@pytest.mark.parametrize('name', list(POINT_SPECS))
def test_point_kernel_exact(cuda_device, name):
    g, m = _fit(name)
    m.e_hat_t_ = torch.as_tensor(np.ravel(g['e_hat'])[None]).to(m.dev_, torch.float64)
    assert _rel(m.sqrt_density(g['Xq']), g['sqrt_density']) <= 1e-11


def test_point_fit_float32(cuda_device):
    g, m = _fit('sinc_dirichlet', np.float32)
    assert _rel(m.predict(g['Xq']), g['predict']) <= 1e-3


def test_point_errors(cuda_device):
    from blml_b200.quick import BLMLQuick
    g = golden('points.npz')['sinc2']
    modes = POINT_SPECS['sinc2'][0]
    with pytest.raises(NotImplementedError):
        BLMLQuick().fit(g['X'], modes, complex_g=True)
    with pytest.raises(ValueError):
        BLMLQuick().fit(g['X'], modes, sample_weight=-np.ones(len(g['X'])))
    m = BLMLQuick(dtype=np.float64, tol=1e-6).fit(g['X'], modes)
    with pytest.raises(ValueError):
        m.predict(np.zeros((3, 3)))


def _point_rows(X, Z, e, kinds, fc, periods):
    import ctypes as C
    import numpy as np
    import torch
    from blml_b200._lib import call
    from blml_b200.binned import point_cols
    d = X.shape[1]
    cols = point_cols({'kinds': list(kinds), 'fc': np.asarray(fc, float), 'periods': list(periods)}, d)
    Xt, Zt, et = (torch.as_tensor(np.ascontiguousarray(a, np.float64)).cuda() for a in (X, Z, e))
    g = torch.empty(len(X), dtype=torch.float64, device='cuda')
    call('blml_point_rows', len(X), d, Xt.data_ptr(), len(Z), Zt.data_ptr(), et.data_ptr(), C.cast(cols, C.c_void_p),
         g.data_ptr(), torch.cuda.current_stream().cuda_stream)
    return g.cpu().numpy()


def test_point_kernel_accuracy(cuda_device):
    """One bin at 0, cut-off 1: g = sin(pi x) / (pi x) against 80-bit arithmetic on an exactly reduced argument, over the
    reduction's range, near zeros, at tiny and at huge arguments. sin is a polynomial of 4e-17 relative error evaluated in
    float64 (its last product and sum round: 1.5 ulp), then pi x and the quotient (1 ulp): 3 2^-53 relative."""
    import numpy as np
    rng = np.random.default_rng(0)
    x = np.concatenate([rng.uniform(-0.5, 0.5, 4000), rng.uniform(-60, 60, 4000), np.arange(1, 50) + 1e-9 * rng.standard_normal(49),
                        10.0 ** rng.uniform(-300, 15, 500), np.arange(-8, 8) / 2 + 0.25, [0.0, 5e-10, 2e-9, 3e15, 2.0 ** 54]])
    g = _point_rows(x[:, None], np.zeros((1, 1)), np.ones(1), ['sinc'], [1.0], [None])
    pi = np.longdouble('3.14159265358979323846264338327950288')
    xl = x.astype(np.longdouble)
    n = np.rint(xl)
    s = np.sin(pi * (xl - n)) * np.where(np.mod(n, 2) == 0, 1, -1)
    ref = np.where(np.abs(x) < 1e-12, 1.0, s / np.where(x == 0, 1, pi * xl))
    assert np.all(np.abs(g - ref) <= 3 * 2.0 ** -53 * np.abs(ref))


@pytest.mark.parametrize('m,B,kinds', [(1, 1, ('sinc',)), (31, 255, ('sinc', 'dirichlet')), (33, 600, ('slits:0.4', 'sinc')),
                                       (200, 5000, ('dirichlet', 'dirichlet:0.5', 'sinc')),
                                       (64, 513, ('sinc',) * 8), (3000, 300, ('ball:0', 'ball:0', 'sinc')), (5, 0, ('sinc',))])
def test_point_kernel_shapes(cuda_device, m, B, kinds):
    """Points and bins around the warp, tile and cluster sizes, on bins (t = 0) and off: the product kernel's sums in
    float64 on the CPU, 1e-13 of sum |terms|. With a ball group the sums are the multi-density kernel's, which takes the
    same Bessel function (CUDA's jn has an absolute error bound, so its tails are not 1e-13 of SciPy's)."""
    import numpy as np
    from blml_b200.local_gpu import point_rows_multi
    from blml_b200.spec import unit_value, units_of
    rng = np.random.default_rng(m + B)
    d = len(kinds)
    X = rng.uniform(-3, 3, (m, d)); Z = rng.uniform(-3, 3, (B, d)); e = rng.standard_normal(B)
    k = min(m, B) // 2
    Z[:k] = X[:k]
    per = [2.5 if kd.startswith('dirichlet') else None for kd in kinds]
    fc = 2.0 + 0.25 * np.arange(d)
    g = _point_rows(X, Z, e, kinds, fc, per)
    K = np.ones((m, B))
    for kind, dims in units_of(list(kinds)):
        K = K * unit_value(kind, fc[dims], [per[j] for j in dims], [X[:, None, j] - Z[None, :, j] for j in dims])
    ref = K @ e
    if any(kd.startswith('ball') for kd in kinds):
        ref = point_rows_multi(X, Z, e[:, None], kinds, fc, per, np.ones((1, len(units_of(list(kinds)))), int))[0][:, 0]
    assert np.all(np.abs(g - ref) <= 1e-13 * (np.abs(K) @ np.abs(e)) + 1e-300)
