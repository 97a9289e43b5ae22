"""Plane-wave sums over a spectrum that starts on an 8-byte boundary: the sums of the same spectrum on a 16-byte one, bit for
bit, at bands of each chunk width (1 to 4 frequencies per lane, several chunks)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('H1,H2,m', [(1, 1, 1), (3, 31, 5), (33, 40, 31), (5, 97, 4), (9, 128, 33), (7, 300, 9)])
def test_spectrum_on_an_8_byte_boundary(cuda_device, H1, H2, m):
    from blml_b200._lib import call
    rng = np.random.default_rng(H1 * H2)
    f1, f2, U = (torch.as_tensor(a).cuda() for a in (np.arange(H1) / 384.0, np.arange(H2) / 400.0, rng.uniform(0, 400, (m, 2))))
    room = torch.zeros(2 * H1 * H2 + 1, dtype=torch.float64, device='cuda')
    spec = torch.as_tensor(rng.standard_normal(2 * H1 * H2)).cuda()
    out = []
    for s in (spec, room[1:]):
        s.copy_(spec)
        g = torch.empty(m, dtype=torch.complex128, device='cuda')
        call('blml_planewave_points', H1, H2, f1.data_ptr(), f2.data_ptr(), s.data_ptr(), m, U.data_ptr(), g.data_ptr(),
             torch.cuda.current_stream().cuda_stream)
        out.append(torch.view_as_real(g))
    assert spec.data_ptr() % 16 == 0 and room[1:].data_ptr() % 16 == 8
    assert torch.isfinite(out[0]).all() and torch.equal(out[0], out[1])
