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
