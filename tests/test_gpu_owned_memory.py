"""Public entries that the Python classes reach through newer forms: groups and runners in the library's own memory
(blml_*_create, blml_lbfgs_batch_set_history) against those in lent memory, and the single-step kernels of the certificate
and the network against their sums and against the fused forms -- the same bits wherever the arithmetic is the same."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _owned(name, *args):
    """The call of a *_create_with entry, made through its form without an allocator."""
    from blml_b200._lib import call
    if name == 'blml_group_create_with':
        return call('blml_group_create', *args[:8], args[-1])
    if name == 'blml_start_batch_create_with':
        return call('blml_start_batch_create', *args[:12], args[-1])
    if name == 'blml_lbfgs_batch_create_with':
        call('blml_lbfgs_batch_create', *args[:13], args[-1])
        if args[13]:
            call('blml_lbfgs_batch_set_history', args[-1]._obj, 1)
        return None
    return call(name, *args)


def _fit(f32, h32, K):
    from blml_b200 import workloads
    from blml_b200.sweep import BLMLBinnedBatch
    rng = np.random.default_rng(0)
    shapes = [(64, 64), (48, 54), (51, 50)]
    counts = [rng.poisson(2.0, s).astype(float) for s in shapes]
    modes = [workloads.pball_modes(s, 0.3) * K for s in shapes]
    init = None if K == 1 else [np.sqrt(c)[None] * np.exp(1j * rng.standard_normal((K,) + s)) for c, s in zip(counts, shapes)]
    b = BLMLBinnedBatch(tol=1e-12, max_sweeps=30, dtype=np.float32 if f32 else np.float64)
    b._history_f32 = h32
    res = b.fit(counts, modes, init=init)
    return b.E_t.cpu().numpy(), np.array([r.loglik_ for r in res]), b.certificate()


@pytest.mark.parametrize('f32,h32,K', [(False, False, 1), (False, False, 2), (False, True, 2), (True, False, 2)])
def test_owned_and_lent_memory_give_the_same_fit(cuda_device, monkeypatch, f32, h32, K):
    from blml_b200 import sweep
    lent = _fit(f32, h32, K)
    monkeypatch.setattr(sweep, 'call', _owned)
    for a, b in zip(lent, _fit(f32, h32, K)):
        assert np.all(np.isfinite(a))
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize('n,np_,col', [(1, 1, 0), (5, 47, 46), (130, 20, -1)])
def test_lanczos_coefficients(cuda_device, n, np_, col):
    from blml_b200._lib import call
    st = torch.cuda.current_stream().cuda_stream
    d = torch.randn(n, np_, dtype=torch.float64, device='cuda')
    coef = torch.empty(n, np_ + 1, dtype=torch.float64, device='cuda')
    alpha = torch.full((n,), 7.0, dtype=torch.float64, device='cuda')
    call('blml_lanczos_coef', n, np_, d.data_ptr(), coef.data_ptr(), alpha.data_ptr(), col, st)
    assert torch.equal(coef, torch.cat([torch.ones_like(d[:, :1]), -d], 1))
    assert torch.equal(alpha, d[:, col] if col >= 0 else torch.full_like(alpha, 7.0))
    q = torch.randn(n, dtype=torch.float64, device='cuda'); q[0] = 0.0
    beta, scale = torch.empty_like(q), torch.empty_like(q)
    call('blml_lanczos_beta', n, q.data_ptr(), beta.data_ptr(), scale.data_ptr(), st)
    want = q.clamp(min=0).sqrt()
    assert torch.equal(beta, want) and torch.equal(scale, torch.where(want > 0, 1 / want, torch.zeros_like(want)))


@pytest.mark.parametrize('N,h,w,C,Cs,c0', [(1, 1, 1, 1, 3, 2), (2, 5, 3, 32, 96, 64)])
def test_upsampling(cuda_device, N, h, w, C, Cs, c0):
    from blml_b200._lib import call
    X = torch.randn(N, h, w, C, device='cuda').to(torch.bfloat16)
    Y = torch.zeros(N, 2 * h, 2 * w, Cs, dtype=torch.bfloat16, device='cuda')
    call('blml_nn_up_fwd', X.data_ptr(), N, h, w, C, Y.data_ptr(), Cs, c0, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(Y[..., c0:c0 + C], X.repeat_interleave(2, 1).repeat_interleave(2, 2))
    Y[..., c0:c0 + C] = 0
    assert not Y.any()


@pytest.mark.parametrize('P,C,Cs', [(1, 8, 8), (300, 32, 96)])
def test_relu_gradient_alone_and_fused(cuda_device, P, C, Cs):
    from blml_b200._lib import call
    st = torch.cuda.current_stream().cuda_stream
    dY = torch.randn(P, Cs, device='cuda'); Y = torch.randn(P, Cs, device='cuda').to(torch.bfloat16)
    c0 = Cs - C
    dpre, fused = (torch.empty(P, C, dtype=torch.bfloat16, device='cuda') for _ in range(2))
    dpreT = torch.empty(C, P, dtype=torch.bfloat16, device='cuda')
    part, db = torch.empty(3, C, device='cuda'), torch.empty(C, device='cuda')
    call('blml_nn_relu_bwd', dY.data_ptr(), Cs, c0, Y.data_ptr(), Cs, c0, P, C, dpre.data_ptr(), dpreT.data_ptr(), st)
    call('blml_nn_relu_bwd_bias', dY.data_ptr(), Cs, c0, Y.data_ptr(), Cs, c0, P, C, fused.data_ptr(), 3, part.data_ptr(),
         db.data_ptr(), st)
    assert torch.equal(dpre, fused) and torch.equal(dpreT, fused.T)


def test_adam_of_one_tensor_and_of_many(cuda_device):
    import ctypes as C
    from blml_b200 import _lib
    from blml_b200._lib import call
    st = torch.cuda.current_stream().cuda_stream
    shapes = [(1,), (33, 70), (1024,), (1025,), (8, 9)] + [(5,)] * 30            # more than one launch takes
    g = torch.Generator(device='cuda').manual_seed(0)
    new = lambda s: torch.randn(s, device='cuda', generator=g)
    one = [dict(w=new(s), g=new(s), m=new(s) * 0.1, v=new(s).square()) for s in shapes]
    many = [{k: t.clone() for k, t in d.items()} for d in one]
    bf = [[(torch.zeros(s, dtype=torch.bfloat16, device='cuda'), torch.zeros(s[::-1], dtype=torch.bfloat16, device='cuda'))
           if len(s) == 2 else (None, None) for s in shapes] for _ in range(2)]
    ptr = lambda t: None if t is None else t.data_ptr()
    for step in (1, 2):
        ts = (_lib.AdamTensor * len(shapes))()
        for i, s in enumerate(shapes):
            r, c = s if len(s) == 2 else (0, 0)
            d = one[i]
            call('blml_nn_adam', *(d[k].data_ptr() for k in 'wgmv'), d['w'].numel(), 1e-3, 0.9, 0.999, 1e-8, step,
                 ptr(bf[0][i][0]), ptr(bf[0][i][1]), r, c, st)
            ts[i].w, ts[i].g, ts[i].m, ts[i].v = (many[i][k].data_ptr() for k in 'wgmv')
            ts[i].n, ts[i].rows, ts[i].cols = d['w'].numel(), r, c
            ts[i].wb, ts[i].wbt = ptr(bf[1][i][0]), ptr(bf[1][i][1])
        call('blml_nn_adam_multi', C.cast(ts, C.c_void_p), len(shapes), 1e-3, 0.9, 0.999, 1e-8, step, st)
        for i in range(len(shapes)):
            assert all(torch.equal(one[i][k], many[i][k]) for k in 'wmv')
            if bf[0][i][0] is not None:
                assert torch.equal(bf[0][i][0], bf[1][i][0]) and torch.equal(bf[0][i][1], bf[1][i][1])
                assert torch.equal(bf[0][i][0], one[i]['w'].to(torch.bfloat16))
                assert torch.equal(bf[0][i][1], one[i]['w'].T.to(torch.bfloat16))
