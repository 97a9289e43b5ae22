"""An L-BFGS runner run a second time, with a shorter cap than the first run's: the fit of a fresh runner with that cap, bit for
bit, whatever pairs the first run left in the memory."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fit(monkeypatch, first, dtype, h32):
    from blml_b200 import sweep, workloads
    from blml_b200._lib import call
    from blml_b200.sweep import BLMLBinnedBatch
    rng = np.random.default_rng(0)
    shapes = [(64, 64), (48, 54), (51, 50)]
    counts = [rng.poisson(2.0, s).astype(float) for s in shapes]
    modes = [workloads.pball_modes(s, 0.3) * 2 for s in shapes]
    init = [np.sqrt(c)[None] * np.exp(1j * rng.standard_normal((2,) + s)) for c, s in zip(counts, shapes)]
    b = BLMLBinnedBatch(tol=1e-12, max_sweeps=3, dtype=dtype)
    b._history_f32 = h32
    device_run = BLMLBinnedBatch._lbfgs_device

    def run(self, E):
        E0 = E.clone()

        def twice(name, *args):
            if name == 'blml_lbfgs_batch_run' and first:
                for cap in (first, 3):
                    caps = np.full(len(shapes), cap, np.int64)
                    call('blml_lbfgs_batch_set_caps', args[0], caps.ctypes.data_as(C.c_void_p))
                    E.copy_(E0)
                    call(name, *args)
                return None
            return call(name, *args)
        monkeypatch.setattr(sweep, 'call', twice)
        try:
            return device_run(self, E)
        finally:
            monkeypatch.setattr(sweep, 'call', call)
    monkeypatch.setattr(BLMLBinnedBatch, '_lbfgs_device', run)
    res = b.fit(counts, modes, init=init)
    monkeypatch.undo()
    return b.E_t.cpu().numpy(), np.array([r.loglik_ for r in res]), b.lbfgs_stats_['iterations']


@pytest.mark.parametrize('dtype,h32', [(np.float64, False), (np.float64, True), (np.float32, False)])
def test_second_run_starts_afresh(cuda_device, monkeypatch, dtype, h32):
    e0, l0, _ = _fit(monkeypatch, 0, dtype, h32)
    e1, l1, steps = _fit(monkeypatch, 30, dtype, h32)
    assert steps >= 30 and np.all(np.isfinite(e0)) and np.all(np.isfinite(e1))
    np.testing.assert_array_equal(l0, l1)
    np.testing.assert_array_equal(e0, e1)
