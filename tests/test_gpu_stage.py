"""The restricted-transform stages (csrc/matvec.cu) on plans of random frequencies and weights against the dense sum in
NumPy: lattices and frequency counts around the tiles of 16 and 32 and the slices of 16, 32 and 64, one to three axes, real and
complex input, batches, sizes on both sides of the tile rules; single plans and groups."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plan(shape, nf, seed, code):
    from blml_b200 import operator as op_mod
    rng = np.random.default_rng(seed)
    freqs = [rng.uniform(-0.5, 0.5, n) for n in nf]
    W = rng.standard_normal(nf)
    return op_mod.Plan(freqs, W, shape, code), freqs, W


def _dense(freqs, W, shape, x):
    V = [np.exp(2j * np.pi * np.outer(np.arange(m), f)) for m, f in zip(shape, freqs)]     # (M, H) per axis
    for a, v in enumerate(V):
        x = np.moveaxis(np.tensordot(x, v.conj(), (a + 1, 0)), -1, a + 1)
    x = x * W
    for a, v in enumerate(V):
        x = np.moveaxis(np.tensordot(x, v, (a + 1, 1)), -1, a + 1)
    return x


CASES = [((1,), (1,), 1), ((5,), (3,), 3), ((1024,), (110,), 1), ((7, 9), (17, 8), 2), ((8, 16), (16, 8), 1),
         ((51, 51), (17, 17), 1), ((33, 65), (31, 64), 5), ((200, 150), (80, 85), 2), ((130, 70), (33, 41), 16),
         ((64, 48), (65, 47), 70), ((130, 140), (129, 120), 80), ((9, 10, 11), (12, 5, 7), 2), ((3, 4, 5, 6), (2, 3, 4, 5), 1)]


@pytest.mark.parametrize('f32', [False, True])
@pytest.mark.parametrize('shape,nf,nb', CASES)
def test_stages_match_dense(cuda_device, shape, nf, nb, f32):
    """Sums of M products per stage, 2 d stages: float64 1e-13 of the largest value, float32 2e-6 per hundred terms."""
    from blml_b200 import _lib
    p, freqs, W = _plan(shape, nf, len(shape) * 100 + nb, _lib.F32 if f32 else _lib.F64)
    rng = np.random.default_rng(1)
    st = torch.cuda.current_stream().cuda_stream
    for cx in (True, False):
        x = rng.standard_normal((nb,) + shape) + (1j * rng.standard_normal((nb,) + shape) if cx else 0)
        dt = (torch.complex64 if cx else torch.float32) if f32 else (torch.complex128 if cx else torch.float64)
        xt = torch.as_tensor(x).cuda().to(dt).contiguous()
        y = torch.empty_like(xt)
        p.apply(xt, y, nb, cx, st)
        ref = _dense(freqs, W, shape, xt.cpu().numpy().astype(complex))
        ref = ref if cx else ref.real
        tol = 2e-6 * max(1.0, max(shape + nf) / 100) if f32 else 1e-13 * len(shape)
        assert np.abs(y.cpu().numpy() - ref).max() <= tol * np.abs(ref).max()


@pytest.mark.parametrize('f32', [False, True])
@pytest.mark.parametrize('many,scale,batch', [(1, 1, 1), (1, 4, 1), (6, 1, 1), (60, 1, 1), (6, 4, 16)])
def test_grouped_stages_equal_single(cuda_device, many, scale, batch, f32):
    """Uneven problems in one group (small, middle and large launches), a subset with one problem off: each problem's
    result is its plan's own (float64: the same sums in the same order whatever the tile), the others stay untouched."""
    from blml_b200 import _lib
    from blml_b200._lib import call
    from blml_b200.sweep import _Group
    code = _lib.F32 if f32 else _lib.F64
    dt = torch.complex64 if f32 else torch.complex128
    sizes = [((scale * (20 + 7 * (g % 5)), scale * (31 + 3 * (g % 7))), (scale * (11 + g % 9), scale * 23), batch * (1 + g % 3))
             for g in range(many)]
    plans = [_plan(s, nf, g, code)[0] for g, (s, nf, _) in enumerate(sizes)]
    nbs = [nb for _, _, nb in sizes]
    off = np.concatenate([[0], np.cumsum([nb * s[0] * s[1] for s, _, nb in sizes])])
    x = torch.randn(int(off[-1]), dtype=dt, device='cuda', generator=torch.Generator(device='cuda').manual_seed(2))
    y = torch.zeros_like(x)
    grp = _Group(plans, x, off[:-1], y, off[:-1], True, nbs)
    assert grp.route == _lib.ROUTE_CONTRACT
    st = torch.cuda.current_stream().cuda_stream
    live = torch.ones(many, dtype=torch.int32, device='cuda')
    sub = torch.arange(many // 3, many, dtype=torch.int32, device='cuda')
    if many > 3:
        live[many // 2] = 0
    call('blml_group_matvec_masked', grp._h, sub.data_ptr(), int(sub.numel()), live.data_ptr(), st)
    for g in range(many):
        a, b = int(off[g]), int(off[g + 1])
        if g < many // 3 or not live[g]:
            assert not y[a:b].any()
            continue
        ref = torch.empty_like(x[a:b])
        plans[g].apply(x[a:b].contiguous(), ref, nbs[g], True, st)
        assert (y[a:b] - ref).abs().max() <= (2e-6 if f32 else 0.0) * ref.abs().max()
