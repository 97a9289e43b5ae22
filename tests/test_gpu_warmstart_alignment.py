"""The learned start's network on views that begin off the boundaries of its wide loads: input of 16 bytes, fields and
targets of 8. The values of aligned copies, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _off(t, by):
    """t's values in a view that starts `by` elements into its storage."""
    room = torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)
    v = room[by:].view(t.shape)
    v.copy_(t)
    return v


def test_forward_and_gradients_of_a_shifted_input(cuda_device):
    from blml_b200.warmstart import WarmStartNet
    g = torch.Generator(device='cuda').manual_seed(0)
    x = torch.randn(2, 16, 24, 8, device='cuda', generator=g).to(torch.bfloat16)
    du = torch.randn(2, 16, 24, 2, device='cuda', generator=g)
    out = []
    for v in (x, _off(x, 1), _off(x, 3)):
        net = WarmStartNet(seed=1)
        u = net.forward(v, 2, 16, 24).clone()
        net.backward(du)
        out.append((u, {k: w.clone() for k, w in net.g.items()}))
        net.check()
    assert _off(x, 1).data_ptr() % 16 == 2
    for u, grads in out[1:]:
        assert torch.equal(u, out[0][0])
        assert all(torch.equal(grads[k], w) for k, w in out[0][1].items())


@pytest.mark.parametrize('HW,S', [(1, 1), (255, 3), (4096, 2)])
def test_loss_of_shifted_fields(cuda_device, HW, S):
    from blml_b200._lib import call
    g = torch.Generator(device='cuda').manual_seed(HW)
    u, t = (torch.randn(S, HW, 2, device='cuda', generator=g) for _ in range(2))
    out = []
    for a, b in ((u, t), (_off(u, 1), t), (u, _off(t, 1)), (_off(u, 1), _off(t, 3))):
        stats = torch.empty(6 * S, dtype=torch.float64, device='cuda'); loss = torch.empty(S, dtype=torch.float64, device='cuda')
        du = torch.empty_like(u)
        call('blml_nn_phase_loss', a.data_ptr(), b.data_ptr(), HW, S, stats.data_ptr(), du.data_ptr(), loss.data_ptr(),
             torch.cuda.current_stream().cuda_stream)
        out.append((stats, loss, du))
    assert _off(u, 1).data_ptr() % 8 == 4
    for got in out[1:]:
        assert all(torch.equal(p, q) for p, q in zip(got, out[0]))
