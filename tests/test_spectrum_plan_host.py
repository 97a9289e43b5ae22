"""What a fit keeps for its predictions (BLMLBinned._spectrum_plan): one entry per kernel, lattice, device and stream, the
oldest dropped -- a fit object that moves to another device or lattice does not meet the former one's plan."""
import types

import numpy as np
import torch

from blml_b200 import _lib
from blml_b200.binned import BLMLBinned
from blml_b200.spec import parse_modes
from blml_b200.workloads import pball_modes


def _fit(monkeypatch, stream):
    monkeypatch.setattr(_lib, 'current_stream', lambda device: stream[0])
    m = BLMLBinned()
    m._code = _lib.F64
    return m


def _place(m, device, shape=(8, 6)):
    """The fit as a fit on `device` leaves it."""
    m.specs_ = parse_modes(pball_modes(shape, 0.3), 2)[0]
    m.shape_, m.d_, m.dev_ = shape, 2, torch.device(device)
    m.h_, m.origin_ = np.ones(2), np.zeros(2)
    plan = types.SimpleNamespace(engine=_lib.ENGINE_SIMT, at=device, shape=shape)
    m.kern_ = [(plan, 1.0, ([np.zeros(3), np.zeros(2)], None))]
    return plan


def test_entry_follows_device_and_stream(monkeypatch):
    stream = [0]
    m = _fit(monkeypatch, stream)
    for device in ('cpu', 'meta', 'cpu'):
        plan = _place(m, device)
        got, _, dev = m._spectrum_plan(0)
        assert got.at == device and all(t.device.type == device for t in dev)
        assert m._spectrum_plan(0)[0] is got and (device == 'cpu' or got is plan)
    first = m._spectrum_plan(0)
    stream[0] = 7
    assert m._spectrum_plan(0) is not first


def test_entries_are_bounded(monkeypatch):
    m = _fit(monkeypatch, [0])
    for i in range(20):
        plan = _place(m, 'cpu', (8, 6 + 2 * i))
        assert m._spectrum_plan(0)[0] is plan and len(m._spec_plans) <= 8
