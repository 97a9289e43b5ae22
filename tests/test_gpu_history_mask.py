"""The L-BFGS runner's history while it fills and after: slots without a pair are not read, whatever their memory holds
(fresh memory full of NaN against fresh memory full of zeros, bit for bit), at memories around the iteration count, for
each storage of the history."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fit(fill, m, iters, dtype, h32, K):
    from blml_b200 import workloads
    from blml_b200.sweep import BLMLBinnedBatch
    torch.cuda.empty_cache()
    dirt = torch.full((1 << 25,), fill, device='cuda', dtype=torch.float64)        # the runner's memory comes from here
    small = [torch.full((1 << 16,), fill, device='cuda', dtype=torch.float64) for _ in range(8)]
    torch.cuda.synchronize()
    del dirt, small
    rng = np.random.default_rng(0)
    shapes = [(64, 64), (48, 54), (51, 50)]
    counts = [rng.poisson(2.0, s).astype(float) for s in shapes]
    modes = [workloads.pball_modes(s, 0.3) * K for s in shapes]
    init = [np.sqrt(c)[None] * np.exp(1j * rng.standard_normal((K,) + s)) for c, s in zip(counts, shapes)]
    b = BLMLBinnedBatch(tol=1e-12, max_sweeps=iters, lbfgs_m=m, dtype=dtype)
    b._history_f32 = h32
    res = b.fit(counts, modes, init=init)
    return np.array([r.loglik_ for r in res]), b.E_t.cpu().numpy()


@pytest.mark.parametrize('dtype,h32', [(np.float64, False), (np.float64, True), (np.float32, False)])
@pytest.mark.parametrize('m,iters', [(1, 4), (3, 2), (3, 3), (3, 8), (9, 20), (20, 6), (20, 45)])
def test_unfilled_slots_are_not_read(cuda_device, m, iters, dtype, h32):
    l0, e0 = _fit(0.0, m, iters, dtype, h32, 2)
    l1, e1 = _fit(float('nan'), m, iters, dtype, h32, 2)
    assert np.all(np.isfinite(l1)) and np.all(np.isfinite(e1))
    np.testing.assert_array_equal(l0, l1)
    np.testing.assert_array_equal(e0, e1)
