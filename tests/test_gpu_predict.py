"""The binned fit at arbitrary points (BLMLBinned.sqrt_density / predict / predict_grid, blml_binned.py:451-500)
against the reference's own values at its own coefficients (tests/golden/predict.npz, made by
tests/golden/make_predict_golden.py): sinc, slits-free sinc rank 2 per mode, dirichlet, sinc x sinc, pball and pball
with a background pball, 2-D ball, 3-D ball (a half-integer Bessel order) and a 2-D ball group times a sinc column;
exact kernels for the interval and radial bands, the harmonic sums for the periodic ones (1e-10 of the largest
value)."""
import numpy as np
import pytest
import torch

from conftest import golden
from golden_cases import FIT_SPECS, PREDICT_EXTRA

pytestmark = pytest.mark.gpu

CASES = ('d1_sinc_real', 'd1_sinc_complex', 'd1_sinc_rank2_permode', 'd1_dir_circ_real', 'd2_sinc_sinc_real',
         'd2_pball_lbfgs', 'd2_pball_bg_lbfgs', 'd2_ball_real') + tuple(PREDICT_EXTRA)


@pytest.mark.parametrize('name', CASES)
def test_points_match_reference(cuda_device, name):
    from blml_b200.binned import BLMLBinned
    g = golden('predict.npz')[name]
    modes, fkw, ckw = PREDICT_EXTRA[name][1:] if name in PREDICT_EXTRA else FIT_SPECS[name]
    kw = dict(ckw); kw['max_sweeps'] = 0
    m = BLMLBinned(dtype=np.float64, device='cuda', **kw).fit(g['counts'], modes, **fkw)
    E = torch.as_tensor(g['e_hat']).reshape(g['e_hat'].shape[0], -1).to('cuda')
    m.e_hat_t_ = E if m.complex_g_ else E.real.contiguous() if E.is_complex() else E
    sd = m.sqrt_density(g['X'])
    ref = g['sqrt_density']
    assert sd.shape == ref.shape
    assert np.abs(sd - ref).max() <= 1e-10 * np.abs(ref).max(), np.abs(sd - ref).max()
    p = m.predict(g['X'])
    assert np.abs(p - g['predict']).max() <= 1e-10 * np.abs(g['predict']).max()
    gr = m.predict_grid(2)
    assert gr.shape == g['grid2'].shape
    assert np.abs(gr - g['grid2']).max() <= 1e-10 * np.abs(g['grid2']).max()


@pytest.mark.parametrize('H1,H2,m', [(1, 1, 1), (3, 31, 5), (33, 32, 31), (64, 65, 33), (5, 97, 4), (31, 129, 70), (40, 300, 9)])
def test_planewave_sizes(cuda_device, H1, H2, m):
    """The plane-wave sum over bands around the lane, chunk and block sizes against the sum in float64 on the CPU; phases
    are reduced exactly, so 1e-13 of sum |C|."""
    import numpy as np
    import torch
    from blml_b200._lib import call
    rng = np.random.default_rng(H1 * H2)
    f1 = np.arange(-(H1 // 2), H1 - H1 // 2) / 384.0; f2 = np.arange(-(H2 // 2), H2 - H2 // 2) / 400.0
    C = rng.standard_normal((H1, H2)) + 1j * rng.standard_normal((H1, H2))
    U = rng.uniform(-10, 400, (m, 2))
    dev = [torch.as_tensor(a).cuda() for a in (f1, f2, C, U)]
    g = torch.empty(m, dtype=torch.complex128, device='cuda')
    call('blml_planewave_points', H1, H2, dev[0].data_ptr(), dev[1].data_ptr(), dev[2].data_ptr(), m, dev[3].data_ptr(),
         g.data_ptr(), torch.cuda.current_stream().cuda_stream)
    p1, p2 = (np.exp(2j * np.pi * (U[:, [a]] * f - np.rint(U[:, [a]] * f))) for a, f in ((0, f1), (1, f2)))
    ref = np.einsum('mi,ij,mj->m', p1, C, p2)
    assert np.all(np.abs(g.cpu().numpy() - ref) <= 1e-13 * np.abs(C).sum())
