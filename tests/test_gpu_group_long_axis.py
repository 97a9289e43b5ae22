"""A group with a 1-D lattice of more points than 65,535 tiles of 32 hold, beside a short one: each plan by itself, bit for bit,
all problems and a subset of one."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('cplx', [True, False])
def test_group_with_a_long_axis(cuda_device, cplx):
    from blml_b200 import _lib, operator as op_mod
    from blml_b200._lib import call
    from blml_b200.sweep import _Group
    rng = np.random.default_rng(0)
    sizes, plans = (2_200_003, 1000), []
    for M, H in zip(sizes, (3, 5)):
        plans.append(op_mod.Plan([rng.uniform(-0.5, 0.5, H)], rng.standard_normal(H), (M,), _lib.F64))
    off = [0, sizes[0]]
    x = torch.randn(sum(sizes), dtype=torch.complex128 if cplx else torch.float64, device='cuda')
    y, ref = torch.zeros_like(x), torch.empty_like(x)
    st = torch.cuda.current_stream().cuda_stream
    for p, o, M in zip(plans, off, sizes):
        p.apply(x[o:o + M], ref[o:o + M], 1, cplx, st)
    g = _Group(plans, x, off, y, off, cplx)
    assert g.route == _lib.ROUTE_CONTRACT
    g(st)
    assert torch.equal(y, ref) and torch.isfinite(torch.view_as_real(y) if cplx else y).all()
    y.zero_()
    one = torch.zeros(1, dtype=torch.int32, device='cuda')
    call('blml_group_matvec_masked', g.on(st), one.data_ptr(), 1, None, st)
    assert torch.equal(y[:sizes[0]], ref[:sizes[0]]) and not y[sizes[0]:].any()
