"""Mat-vecs launched behind the kernel that writes their input (programmatic dependent launches): a chain whose every input
is the output of the launch before, or of an elementwise kernel, against the same chain with the device idle between the
links, bit for bit. One-launch clusters, three-launch FFTs, restricted transforms, a few plans in one chain, groups."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LINKS = 12


def _plan(shape, fc, code, route):
    from blml_b200 import operator as op_mod, _lib, workloads
    from blml_b200.spec import parse_modes
    sp, _ = parse_modes(workloads.pball_modes(shape, fc), 2)
    p = op_mod.Plan(*op_mod.mode_transform(sp[0], shape, np.ones(2), shape), shape, code, _lib.ENGINE_SIMT)
    p.route = route
    return p


def _types(f64, cplx):
    return {(True, True): torch.complex128, (True, False): torch.float64,
            (False, True): torch.complex64, (False, False): torch.float32}[f64, cplx]


def _chain(x, scale, apply, wait):
    """LINKS times x <- S (scale x) through two buffers; every intermediate is returned."""
    a, b, out = x.clone(), torch.empty_like(x), []
    for _ in range(LINKS):
        a.mul_(scale)
        if wait:
            torch.cuda.synchronize()
        apply(a, b)
        if wait:
            torch.cuda.synchronize()
        out.append(b.clone())
        if wait:
            torch.cuda.synchronize()
        a, b = b, a
        apply(a, b)                                       # straight behind the launch that wrote a
        a, b = b, a
    return out


def _check(x, apply):
    x1, x2 = torch.empty_like(x), torch.empty_like(x)
    apply(x, x1); apply(x1, x2)
    scale = float(x1.abs().max() / x2.abs().max()) ** 2        # two mat-vecs a link: values stay of order one
    x = x / x.abs().max()
    for got, ref in zip(_chain(x, scale, apply, False), _chain(x, scale, apply, True)):
        assert torch.equal(torch.view_as_real(got) if got.is_complex() else got,
                           torch.view_as_real(ref) if ref.is_complex() else ref)


@pytest.mark.parametrize('f64', [True, False])
@pytest.mark.parametrize('cplx', [True, False])
@pytest.mark.parametrize('shape,nb', [((64, 64), 1), ((81, 64), 2), ((96, 81), 7), ((256, 256), 2), ((243, 162), 3)])
@pytest.mark.parametrize('route', [1, 2])
def test_chained_matvecs(cuda_device, route, shape, nb, cplx, f64):
    from blml_b200 import _lib
    p = _plan(shape, 0.3, _lib.F64 if f64 else _lib.F32, route)
    x = torch.randn((nb,) + shape, dtype=_types(f64, cplx), device='cuda')
    st = torch.cuda.current_stream().cuda_stream
    _check(x, lambda a, b: p.apply(a, b, nb, cplx, st))


@pytest.mark.parametrize('f64', [True, False])
def test_chained_few_plans(cuda_device, f64):
    from blml_b200 import _lib
    from blml_b200._lib import call
    code = _lib.F64 if f64 else _lib.F32
    ps = [_plan((192, 162), fc, code, 2) for fc in (0.1, 0.3)]
    plans = (ctypes.c_void_p * 2)(*[p._h.value for p in ps]); nb = (ctypes.c_int * 2)(1, 1)
    need = int(_lib.lib().blml_matvecs_workspace(2, plans, nb))
    ws = torch.empty(need, dtype=torch.uint8, device='cuda')
    st = torch.cuda.current_stream().cuda_stream
    x = torch.randn((2, 192, 162), dtype=_types(f64, True), device='cuda')
    _check(x, lambda a, b: call('blml_matvecs', 2, plans, nb, a.data_ptr(), b.data_ptr(), 1, ws.data_ptr(), need, st))


@pytest.mark.parametrize('f64', [True, False])
@pytest.mark.parametrize('route', [1, 2])
def test_chained_groups(cuda_device, route, f64):
    from blml_b200 import _lib
    from blml_b200.sweep import _Group
    code = _lib.F64 if f64 else _lib.F32
    shapes = [(64, 64), (96, 81), (128, 54), (256, 192), (72, 72)]
    plans = [_plan(s, 0.25, code, 0) for s in shapes]
    off = np.concatenate([[0], np.cumsum([s[0] * s[1] for s in shapes])])
    x = torch.randn(int(off[-1]), dtype=_types(f64, True), device='cuda')
    st = torch.cuda.current_stream().cuda_stream
    groups = {}

    def apply(a, b):
        key = a.data_ptr(), b.data_ptr()
        if key not in groups:
            groups[key] = _Group(plans, a, off[:-1], b, off[:-1], True)
            groups[key].route = route
        groups[key](st)

    _check(x, apply)
