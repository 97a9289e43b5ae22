"""Memory that groups, batch fits and certificates borrow goes back to torch's allocator when they are done, with Python's
cyclic collector off, and does not reach other work before their own launches are done with it."""
import gc

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def no_gc():
    gc.collect()
    on = gc.isenabled()
    gc.disable()
    yield
    if on:
        gc.enable()


def _batch():
    from blml_b200 import workloads
    rng = np.random.default_rng(0)
    shapes = [(64, 64), (48, 64), (51, 50)]
    return [rng.poisson(3.0, s).astype(float) for s in shapes], [workloads.pball_modes(s, 0.3) for s in shapes]


def _group(nb):
    from blml_b200 import _lib, workloads
    from blml_b200.spec import parse_modes
    from blml_b200.sweep import BLMLBinnedBatch, _Group
    sp, _ = parse_modes(workloads.pball_modes((64, 64), 0.3), 2)
    p, _ = BLMLBinnedBatch()._plan(sp[0], (64, 64), _lib.F64)
    x = torch.randn(nb, 64, 64, dtype=torch.complex128, device='cuda')
    y = torch.empty_like(x); ref = torch.empty_like(x)
    p.apply(x, ref, nb, True, torch.cuda.current_stream().cuda_stream)
    off = [i * 4096 for i in range(nb)]
    return _Group([p] * nb, x, off, y, off, True), x, y, ref


def test_fit_and_certificate_give_back_what_they_borrow(cuda_device, no_gc):
    from blml_b200.sweep import BLMLBinnedBatch
    counts, modes = _batch()
    batch = BLMLBinnedBatch(tol=1e-9, max_sweeps=6)
    batch.fit(counts, modes)
    batch.certificate()
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    for _ in range(3):                                    # the fit's own arrays are replaced, its runners' memory is back
        batch.fit(counts, modes)
        batch.certificate()
        torch.cuda.synchronize()
        assert torch.cuda.memory_allocated() == held


def test_group_gives_back_what_it_borrows(cuda_device, no_gc):
    g, x, y, ref = _group(3)
    held = torch.cuda.memory_allocated()
    lent = sum(t.numel() for t in g._mem.tensors)
    g(torch.cuda.current_stream().cuda_stream)
    del g
    assert lent >= 3 * 4096 * 16 and torch.cuda.memory_allocated() <= held - lent
    torch.testing.assert_close(y, ref, rtol=1e-13, atol=0)


def test_memory_of_a_group_pending_on_another_stream_is_not_reused(cuda_device, no_gc):
    g, x, y, ref = _group(3)
    sizes = [t.numel() for t in g._mem.tensors]
    y.fill_(float('nan'))
    # blocks of these sizes in torch's cache (a new allocation would wait for the device)
    warm = [torch.zeros(n, dtype=torch.uint8, device='cuda') for n in sizes for _ in range(4)]
    del warm
    torch.cuda.synchronize()
    held = torch.cuda.memory_allocated()
    other = torch.cuda.Stream()
    with torch.cuda.stream(other):
        torch.cuda._sleep(400_000_000)                    # about 0.2 s: the launch is still to come when its memory goes back
    g(other.cuda_stream)
    del g
    assert torch.cuda.memory_allocated() <= held - sum(sizes)
    # zeros: descriptors that they replaced would leave the launch without work, and y as it is
    taken = [torch.zeros(n, dtype=torch.uint8, device='cuda') for n in sizes for _ in range(4)]
    torch.cuda.current_stream().synchronize()
    assert not other.query() and len(taken) == 4 * len(sizes)         # (the test's premise)
    torch.cuda.synchronize()
    torch.testing.assert_close(y, ref, rtol=1e-13, atol=0)


@pytest.mark.parametrize('own', [False, True])
def test_group_inside_a_stream_capture(cuda_device, own):
    """A group made on the default stream, captured on a stream of its own and replayed on new input (own: made on the
    capturing stream)."""
    st = torch.cuda.Stream()
    with torch.cuda.stream(st) if own else torch.cuda.stream(torch.cuda.current_stream()):
        g, x, y, ref = _group(3)
    g((st if own else torch.cuda.current_stream()).cuda_stream)
    torch.cuda.synchronize()
    torch.testing.assert_close(y, ref, rtol=1e-13, atol=0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        g(st.cuda_stream)
    x.mul_(2.0)
    y.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    torch.testing.assert_close(y, 2.0 * ref, rtol=1e-13, atol=0)
