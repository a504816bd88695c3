"""Resident 3-D runs (all steps in one launch, fields in shared memory) against the
launch-by-launch kernel, through the C ABI: the same fields, curl records and probe
series bit for bit, the same monitor sums up to the order of their FP64 additions."""

from __future__ import annotations

import ctypes

import pytest
import torch
from conftest import rel_l2

from diffnano_b200 import _lib
from diffnano_b200.solvers import _setup
from diffnano_b200.solvers._engine import Engine, MonitorSpec

REF, PHYS = _lib.DN_AXES_REFERENCE, _lib.DN_AXES_PHYSICAL


def _engine(shape, axes, T, src=None, comp=_lib.DN_EZ, monitors=(), probe=None,
            dtype=torch.float32):
    s = {"type": "gaussian_pulse", "spread": 60.0, "t0": 80.0, **(src or {})}
    eng = Engine(is3d=True, shape=shape, dl=20.0, dt=8.0, pml_layers=min(2, min(shape) // 2),
                 dtype=dtype, device=torch.device("cuda", 0), n_steps=T,
                 wave=_setup.waveform_table(T, 8.0, 0.1, s),
                 src_box=None if src is None else _setup.source_box_3d(shape, s),
                 src_comp=_lib.DN_NONE if src is None else comp, monitors=monitors, probe=probe,
                 axes=axes)
    g = torch.Generator().manual_seed(sum(shape))
    eng.set_eps(1.5 + 2.0 * torch.rand(shape, dtype=torch.float64, generator=g))
    eng.state0 = torch.randn(6, *shape, dtype=torch.float64, generator=g)
    return eng


def _bytes(eng):
    return int(_lib.lib().dn_fdtd3d_workspace_bytes(
        ctypes.byref(eng.grid), ctypes.byref(eng.src), eng.mon_arr, len(eng.monitors),
        eng.n_steps))


def _run(eng, ws_bytes, record):
    """Fields, curls, probe series, monitor sums with a workspace of so many bytes."""
    eng.reset()
    W, T = eng.shape3[2], eng.n_steps
    eng.A[..., :W] = eng.state0.to(eng.device, eng.dtype)
    eng._ws = torch.full((ws_bytes,), 1, dtype=torch.uint8, device=eng.device)
    buf = eng.curl_buffer(T) if record else None
    eng.run(0, T, record=eng.curl_record(buf, 0, T) if record else None)
    eng.check_status()
    same = [eng.field(c).clone() for c in range(6)]
    same += [buf[..., :W]] if record else []
    same += [] if eng.probe_out is None else [eng.probe_out.clone()]
    return same, [a.clone() for a in eng.accs]


def _compare(eng, record=False):
    n = _bytes(eng)
    assert n > 0
    a, sa = _run(eng, n, record)
    b, sb = _run(eng, 0, record)
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    for x, y in zip(sa, sb):
        # two orders of T additions each
        assert float(y.abs().max()) > 0 and rel_l2(x, y) < 4 * eng.n_steps * 2.0 ** -53


# one cell, rows of 1 .. 4 columns past a multiple of four, blocks of one row, blocks
# of unequal sizes, one block, the whole chip, nearly all its shared memory, rows so
# long that the threads hold few of them
SHAPES = [(1, 1, 1), (3, 1, 6), (1, 7, 5), (9, 10, 11), (20, 30, 41), (5, 50, 90), (149, 3, 8),
          (2, 200, 31), (4, 3, 1400), (40, 40, 224), (90, 88, 92)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("record", [False, True])
def test_fields_from_a_random_state(cuda, shape, record):
    for T in (9, 12):  # odd and even: the result ends in either set
        _compare(_engine(shape, PHYS, T), record)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [4, 13, 64, 90])
def test_reference_axes(cuda, n):
    _compare(_engine((n, n, n), REF, 30, src={}), record=True)


@pytest.mark.gpu
@pytest.mark.parametrize("axes", [REF, PHYS])
@pytest.mark.parametrize("src", [{"pos": [3, 20, 39]}, {"plane": "xy"}, {"plane": "yz"}, {}])
def test_sources_monitors_and_probe(cuda, axes, src):
    shape = (40, 40, 40)
    wl = (1550.0, 1310.0)
    mons = [MonitorSpec("a", _lib.DN_EZ, ((7, 8), (0, 40), (0, 40)), wl),
            MonitorSpec("b", _lib.DN_HY, ((0, 40), (3, 5), (1, 38)), wl[:1]),
            MonitorSpec("c", _lib.DN_EX, ((5, 9), (2, 4), (11, 12)), wl)]
    for comp in (_lib.DN_EX, _lib.DN_EY, _lib.DN_EZ):
        _compare(_engine(shape, axes, 40, src, comp, mons, (_lib.DN_HX, (6, 7, 39))), record=True)


@pytest.mark.gpu
def test_samples_beyond_the_workspace_run_in_pieces(cuda):
    """A monitor whose samples of the whole run do not fit in 64 MB."""
    shape, T = (48, 48, 48), 310
    mons = [MonitorSpec("a", _lib.DN_EY, ((0, 48), (0, 48), (0, 48)), (1550.0,))]
    eng = _engine(shape, PHYS, T, {"pos": [20, 20, 20]}, monitors=mons)
    assert 48 ** 3 * 4 * T > 64 << 20
    _compare(eng)


@pytest.mark.gpu
def test_what_stays_launch_by_launch(cuda):
    """Double precision, sources in H, short runs and grids beyond the chip's shared
    memory ask for no workspace; with too small a one a run still gives its result."""
    assert _bytes(_engine((20, 20, 20), PHYS, 20, dtype=torch.float64)) == 0
    assert _bytes(_engine((20, 20, 20), PHYS, 20, {}, _lib.DN_HX)) == 0
    assert _bytes(_engine((20, 20, 20), PHYS, 7)) == 0
    assert _bytes(_engine((128, 128, 128), PHYS, 20)) == 0
    eng = _engine((20, 20, 20), PHYS, 20, {})
    a, _ = _run(eng, _bytes(eng) - 16, False)
    b, _ = _run(eng, _bytes(eng), False)
    assert all(torch.equal(x, y) for x, y in zip(a, b))
