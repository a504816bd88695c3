"""How much memory curl records may take: the share that all live records have in
common, the room left beside them, and the way back to checkpoints."""

from __future__ import annotations

import gc

import pytest
import torch
from test_full_record import _gradient, _solver3d

from diffnano_b200.solvers import _records, fom_abs2
from diffnano_b200.solvers._engine import Engine
from diffnano_b200.solvers.batch2d import BatchInstance, FDTDBatch2D

GB = 1 << 30


class _Props:
    total_memory = 160 * GB


@pytest.fixture
def gpu(monkeypatch):
    """A GPU of 160 GB with 100 GB free, as the allocator would describe it."""
    state = {"free": 90 * GB, "reserved": 15 * GB, "allocated": 5 * GB}
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: _Props)
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda d: (state["free"], 160 * GB))
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict", lambda d: {
        f"{k}_bytes": {"all": {"current": state[k]}} for k in ("reserved", "allocated")})
    return state


def test_live_records_share_an_eighth_of_the_memory(gpu):
    made = []

    def claim(nbytes, device="a"):
        return _records.claim(device, nbytes, 0, lambda: made.append(nbytes) or len(made))

    a = claim(12 * GB)
    assert a.made == 1 and claim(9 * GB) is None and made == [12 * GB]
    b = claim(8 * GB)
    assert b is not None and claim(1) is None
    assert claim(20 * GB, "b") is not None  # another GPU has a share of its own
    del a
    gc.collect()
    assert claim(12 * GB) is not None and claim(21 * GB) is None


def test_a_record_takes_at_most_half_of_what_is_free(gpu):
    gpu["free"] = 15 * GB  # 25 GB with the allocator's reserve of 10
    assert _records.claim("c", 12 * GB, 0, lambda: 1) is not None
    assert _records.claim("d", 12 * GB, GB, lambda: 1) is None
    assert _records.claim("e", 13 * GB, 0, lambda: 1) is None
    gpu["free"] = 0  # the reserve alone is there for the asking
    assert _records.claim("i", 9 * GB, GB, lambda: 1) is not None
    assert _records.claim("j", 10 * GB, GB, lambda: 1) is None


def test_small_records_do_not_ask_what_is_free(gpu):
    gpu["free"] = gpu["reserved"] = gpu["allocated"] = 0
    a = _records.claim("g", GB, 0, lambda: 1)
    b = _records.claim("g", 3 * GB // 2, 0, lambda: 1)  # 2.5 GB in all, a 64th
    assert a and b and _records.claim("g", GB, 0, lambda: 1) is None
    assert _records.claim("h", 3 * GB, 0, lambda: 1) is None


def test_no_record_when_it_cannot_be_allocated(gpu):
    def fail():
        raise torch.OutOfMemoryError("no room")

    assert _records.claim("f", GB, 0, fail) is None
    assert _records.claim("f", 20 * GB, 0, lambda: 1) is not None  # and nothing is counted


@pytest.mark.gpu
def test_several_solves_before_one_backward(cuda, monkeypatch):
    """Room for one record: the first solve keeps it, the second goes by checkpoints,
    and a solve after the backward has it again; every gradient is the same."""
    g = torch.Generator().manual_seed(3)
    eps = [(1.5 + 2.0 * torch.rand(24, 20, 36, dtype=torch.float64, generator=g)).to(cuda)
           for _ in range(3)]
    src = {"type": "gaussian_pulse", "plane": "xy", "z": 7, "component": "Ex"}
    want = [_gradient(_solver3d(cuda), e, src)[1] for e in eps]
    one = 3 * 37 * 24 * 20 * 64 * 4  # record of a solve: 37 steps, rows padded to 64
    gc.collect()
    total = torch.cuda.get_device_properties(cuda).total_memory
    monkeypatch.setattr(_records, "RECORD_SHARE", 1.5 * one / total)
    real, asked = Engine.curl_buffer, []
    monkeypatch.setattr(Engine, "curl_buffer", lambda s, n: asked.append(n) or real(s, n))
    solver, loss, ins = _solver3d(cuda), 0.0, []
    for e in eps[:2]:
        x = e.clone().requires_grad_(True)
        r = solver.forward(x, source=dict(src))
        loss = loss + fom_abs2(r.metadata["monitors"][0]["dft"]) + (r.field.double() ** 2).sum()
        ins.append(x)
    assert asked == [37]  # (a record, then none)
    got = torch.autograd.grad(loss, ins)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert len(asked) == 2 and asked[1] < 37  # a segment's curl terms
    del r, loss
    assert torch.equal(_gradient(solver, eps[2], src)[1], want[2]) and asked[2] == 37


@pytest.mark.gpu
def test_checkpoints_on_a_gpu_that_is_nearly_full(cuda, monkeypatch):
    spec = BatchInstance(grid_shape=(40, 45), n_steps=60, pml_layers=4,
                         source={"type": "gaussian_pulse", "row": 10, "spread": 300.0, "t0": 300.0},
                         monitor={"row": 30, "wavelengths_nm": [1550.0]})
    g = torch.Generator().manual_seed(5)
    eps = [(1.5 + 2.0 * torch.rand(40, 45, dtype=torch.float64, generator=g)).to(cuda)
           for _ in range(3)]

    def run():
        x = [e.clone().requires_grad_(True) for e in eps]
        b = FDTDBatch2D([spec] * 3, "TM", torch.float64, cuda, tile_rows=16)
        _, dfts = b.forward(x)
        return b, torch.autograd.grad(sum((d.abs() ** 2).sum() for d in dfts), x)

    b, want = run()
    assert b.uses_resident(True, True) and b.uses_resident(False, True)
    b._build(False)  # a batch that stops differentiating gives its record back
    assert b._record is None
    monkeypatch.setattr(_records, "UNASKED_SHARE", 0.0)
    monkeypatch.setattr(_records, "is_room", lambda d, n: n <= 60 * 3 * 40 * 64 * 8)
    b, got = run()
    assert not b.uses_resident(True, True) and b.uses_resident(True, False)
    for x, y in zip(got, want):
        assert float((x - y).norm() / y.norm()) < 1e-12
