"""The implicit-GEMM convolutions of the warm start against the explicit form (im2col, GEMM, bias, ReLU) of the same
library on the same inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(name, *a):
    from blml_b200._lib import call
    call(name, *[x.data_ptr() if isinstance(x, torch.Tensor) else x for x in a], torch.cuda.current_stream().cuda_stream)


def _layer(N, H, W, C, Co, Cs, c0, seed=0):
    g = torch.Generator(device='cuda').manual_seed(seed)
    X = torch.randn(N, H, W, Cs, device='cuda', generator=g).to(torch.bfloat16)
    Wt = (torch.randn(Co, 9 * C, device='cuda', generator=g) / (3 * C ** 0.5)).to(torch.bfloat16)
    return g, X, Wt


# the network's layers (8, 32, 64, 96 = 3 x 32, 128, 192, 384 channels), patches that are cut by every side of the
# lattice, lattices smaller than a patch, several images in one patch
@pytest.mark.parametrize('N,H,W,C,Co,Cs,c0,up', [(2, 16, 24, 8, 32, 8, 0, False), (1, 8, 8, 32, 64, 96, 64, True),
                                                 (3, 6, 7, 64, 64, 192, 128, False), (1, 40, 33, 96, 32, 96, 0, True),
                                                 (5, 3, 5, 128, 256, 128, 0, False), (1, 1, 1, 192, 16, 192, 0, True),
                                                 (2, 130, 9, 384, 128, 384, 0, False)])
def test_conv_equals_im2col_gemm(cuda_device, N, H, W, C, Co, Cs, c0, up):
    """Same products in the same order (tap by tap, channels ascending, FP32 accumulation): equal bit for bit."""
    g, X, Wt = _layer(N, H, W, C, Co, Cs, c0)
    bias = torch.randn(Co, device='cuda', generator=g)
    P = N * H * W
    err = torch.zeros(1, dtype=torch.int32, device='cuda')
    Ys, y0 = Co + 16, 8
    Y = torch.zeros(N, H, W, Ys, dtype=torch.bfloat16, device='cuda')
    U = torch.zeros(N, 2 * H, 2 * W, Co + 8, dtype=torch.bfloat16, device='cuda')
    _call('blml_nn_conv3x3', X, N, H, W, Cs, c0, C, Wt, bias, 1, Co, Y, Ys, y0, U if up else None, Co + 8, 8, err)
    col = torch.empty(P, 9 * C, dtype=torch.bfloat16, device='cuda')
    Cm = torch.empty(P, Co, device='cuda')
    ref = torch.zeros_like(Y)
    _call('blml_nn_im2col', X, N, H, W, Cs, c0, C, col, 0)
    _call('blml_nn_gemm_bf16', col, Wt, Cm, P, Co, 9 * C, 1, err)
    _call('blml_nn_bias_act', Cm, 1, P, Co, bias, 1, ref, Ys, y0)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(Y, ref)
    if up:
        want = ref[..., y0:y0 + Co].repeat_interleave(2, 1).repeat_interleave(2, 2)
        assert torch.equal(U[..., 8:], want) and not U[..., :8].any()


@pytest.mark.parametrize('N,H,W,C,Co,Xs,x0', [(1, 8, 8, 32, 32, 96, 64), (3, 6, 7, 64, 64, 64, 0),
                                              (1, 40, 33, 96, 32, 96, 0), (5, 3, 5, 128, 256, 384, 256),
                                              (1, 1, 1, 192, 64, 192, 0), (2, 130, 9, 384, 128, 384, 0)])
def test_dgrad_equals_gemm_col2im(cuda_device, N, H, W, C, Co, Xs, x0):
    """Each tap's product accumulated apart and added in tap order, as the gather over the P x 9C matrix does: equal bit
    for bit."""
    g, D, _ = _layer(N, H, W, Co, Co, Co, 0, seed=1)
    Wt = (torch.randn(9 * C, Co, device='cuda', generator=g) / (3 * Co ** 0.5)).to(torch.bfloat16)
    P = N * H * W
    err = torch.zeros(1, dtype=torch.int32, device='cuda')
    dX = torch.zeros(N, H, W, Xs, device='cuda')
    ref = torch.zeros_like(dX)
    _call('blml_nn_conv3x3_dgrad', D, N, H, W, Co, Wt, C, dX, Xs, x0, err)
    dcol = torch.empty(P, 9 * C, device='cuda')
    _call('blml_nn_gemm_bf16', D, Wt, dcol, P, 9 * C, Co, 1, err)
    _call('blml_nn_col2im', dcol, N, H, W, C, ref, Xs, x0)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(dX, ref)


# rows of 64 pixels and more, of a divisor of 64, of odd and even others; the last block of pixels short
@pytest.mark.parametrize('N,H,W,C,Co,Cs,c0,splits', [(2, 16, 24, 8, 32, 8, 0, 3), (1, 8, 8, 32, 64, 96, 64, 1),
                                                     (3, 8, 7, 64, 64, 192, 128, 4), (1, 40, 34, 96, 32, 96, 0, 20),
                                                     (8, 3, 5, 128, 256, 128, 0, 2), (1, 2, 4, 192, 32, 192, 0, 1),
                                                     (2, 12, 192, 384, 128, 384, 0, 5), (4, 4, 4, 256, 64, 256, 0, 1)])
def test_wgrad_equals_gemm(cuda_device, N, H, W, C, Co, Cs, c0, splits):
    """The transposed im2col matrix and the plain GEMM over the pixels: the same products in the same order and splits
    (the operands' roles swapped), equal bit for bit."""
    g, X, _ = _layer(N, H, W, C, Co, Cs, c0, seed=2)
    D = torch.randn(N, H, W, Co, device='cuda', generator=g).to(torch.bfloat16)
    P = N * H * W
    err = torch.zeros(1, dtype=torch.int32, device='cuda')
    part, pref = (torch.empty(splits, Co, 9 * C, device='cuda') for _ in range(2))
    dW, ref = (torch.empty(Co, 9 * C, device='cuda') for _ in range(2))
    _call('blml_nn_conv3x3_wgrad', X, N, H, W, Cs, c0, C, D, Co, splits, part, dW, err)
    colT = torch.empty(9 * C, P, dtype=torch.bfloat16, device='cuda')
    _call('blml_nn_im2col', X, N, H, W, Cs, c0, C, colT, 1)
    _call('blml_nn_gemm_bf16', D.reshape(P, Co).T.contiguous(), colT, pref, Co, 9 * C, P, splits, err)
    _call('blml_nn_sum_splits', pref, splits, Co * 9 * C, ref)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    assert torch.equal(part, pref) and torch.equal(dW, ref)


@pytest.mark.parametrize('P,C,Cs', [(1, 8, 8), (300, 32, 96), (5000, 256, 256)])
def test_relu_bwd_bias(cuda_device, P, C, Cs):
    g = torch.Generator(device='cuda').manual_seed(3)
    dY = torch.randn(P, Cs, device='cuda', generator=g)
    Y = torch.randn(P, Cs, device='cuda', generator=g).to(torch.bfloat16)
    c0 = Cs - C
    dpre = torch.empty(P, C, dtype=torch.bfloat16, device='cuda')
    chunks = 7
    part = torch.empty(chunks, C, device='cuda')
    db = torch.empty(C, device='cuda')
    _call('blml_nn_relu_bwd_bias', dY, Cs, c0, Y, Cs, c0, P, C, dpre, chunks, part, db)
    want = torch.where(Y[:, c0:] > 0, dY[:, c0:], torch.zeros_like(dY[:, c0:]))
    assert torch.equal(dpre, want.to(torch.bfloat16))
    ref = torch.empty_like(db)                   # the bias gradient on its own: the same sums in the same order
    _call('blml_nn_bias_grad', dY, Cs, c0, Y, Cs, c0, P, C, 1, chunks, part, ref)
    assert torch.equal(db, ref)


@pytest.mark.parametrize('P,chunks', [(1, 1), (1000, 7), (70000, 64)])
def test_head_gradients(cuda_device, P, chunks):
    """dY^T X and the column sums of dY in float64; FP32 sums of P products, chunk by chunk."""
    g = torch.Generator(device='cuda').manual_seed(4)
    X = torch.randn(P, 32, device='cuda', generator=g).to(torch.bfloat16)
    dY = torch.randn(P, 2, device='cuda', generator=g)
    Wt = torch.randn(2, 32, device='cuda', generator=g)
    part = torch.empty(chunks, 66, device='cuda')
    gw, dX = torch.empty(2, 33, device='cuda'), torch.empty(P, 32, device='cuda')
    _call('blml_nn_head_bwd', dY, X, P, 32, 2, Wt, dX, chunks, part, gw)
    ref = torch.cat([dY.double().T @ X.double(), dY.double().sum(0)[:, None]], 1)
    top = dY.abs().max().item() * X.float().abs().max().item()
    assert (gw - ref).abs().max().item() <= (P / chunks + chunks + 2) * 2.0 ** -24 * P ** 0.5 * top
