"""blml_matvecs: several plans on consecutive lattices in one call against each plan's own mat-vec, bit for bit -- FFT
routes in one launch chain, small lattices (a chain of their own), contraction routes, mixed ones, more than a chain
holds, real and complex, both types."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [((256, 256), [.33, .05], [1, 1]), ((256, 256), [.33, .05, .2, .4], [1, 2, 3, 1]), ((144, 162), [.1, .45], [2, 5]),
         ((64, 64), [.3, .1], [1, 1]), ((64, 64), [.3, .1], [40, 1]), ((200, 192), [.3, .1], [1, 1]),
         ((256, 128), [.3, .2, .1, .05, .4], [1, 1, 1, 1, 1]), ((51, 50), [.3, .1], [2, 1])]


@pytest.mark.parametrize('f32', [False, True])
@pytest.mark.parametrize('cx', [True, False])
@pytest.mark.parametrize('shape,fcs,nb', CASES)
def test_matvecs_equal_each_plan(cuda_device, shape, fcs, nb, cx, f32):
    from blml_b200 import _lib, workloads
    from blml_b200.operator import Plan, mode_transform, pad_rule
    from blml_b200.spec import parse_modes
    h = np.ones(2)
    plans = []
    for fc in fcs:
        sp, _ = parse_modes(workloads.pball_modes(shape, fc), 2)
        plans.append(Plan(*mode_transform(sp[0], shape, h, pad_rule(shape, h, sp)), shape, _lib.F32 if f32 else _lib.F64))
    dt = {(True, True): torch.complex64, (True, False): torch.complex128, (False, True): torch.float32,
          (False, False): torch.float64}[cx, f32]
    x = torch.randn((sum(nb),) + shape, dtype=dt, device='cuda', generator=torch.Generator(device='cuda').manual_seed(1))
    y = torch.empty_like(x); ref = torch.empty_like(x)
    st = torch.cuda.current_stream().cuda_stream
    at = 0
    for p, n in zip(plans, nb):
        p.apply(x[at:at + n], ref[at:at + n], n, cx, st)
        at += n
    hs = (ctypes.c_void_p * len(plans))(*[p._h.value for p in plans])
    ns = (ctypes.c_int * len(nb))(*nb)
    need = _lib.lib().blml_matvecs_workspace(len(plans), hs, ns)
    ws = torch.empty(max(need, 1), dtype=torch.uint8, device='cuda')
    with pytest.raises(_lib.BLMLError):
        _lib.call('blml_matvecs', len(plans), hs, ns, x.data_ptr(), y.data_ptr(), int(cx), ws.data_ptr(), need - 1, st)
    _lib.call('blml_matvecs', len(plans), hs, ns, x.data_ptr(), y.data_ptr(), int(cx), ws.data_ptr(), need, st)
    assert torch.equal(y, ref)
