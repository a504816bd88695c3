"""How resident runs are planned (on the host, for a GPU of 148 multiprocessors), and
runs whose monitor samples need several launches."""

from __future__ import annotations

import ctypes

import pytest
import torch
from conftest import rel_l2
from test_resident2d import _compare, _compare_sweeps, _comps, _engine, _run, _sweep, _tol
from test_resident3d import _compare as _compare3d
from test_resident3d import _engine as _engine3d

from diffnano_b200 import _lib
from diffnano_b200.solvers._engine import MonitorSpec
from oracle import fdtd_ref as R

SMS = 148
TM, TE, F32, F64 = _lib.DN_TM, _lib.DN_TE, torch.float32, torch.float64


def plan2d(H, W, steps, pol=TM, dtype=F32, cells=(0, 0), adjoint=False):
    """Plan of a solve with a monitor over the first cells[0] x cells[1] cells."""
    g = _lib.DnGrid(D=1, H=H, W=W, dtype=_lib.DN_F32 if dtype == F32 else _lib.DN_F64,
                    pitch_y=(W + 31) // 32 * 32, pitch_z=H * ((W + 31) // 32 * 32), dt=7.0, dl=20.0,
                    axes=0, pol=pol)
    mon = _lib.DnMonitor(component=_lib.DN_EZ if pol == TM else _lib.DN_HZ, n_freq=1,
                         box=_lib.box((0, 0, 0), (1, *cells)))
    out = _lib.DnResidentPlan()
    _lib.check("plan", _lib.lib().dn_fdtd2d_resident_plan(
        ctypes.byref(g), None, ctypes.byref(mon), int(cells[0] > 0), steps, int(adjoint), SMS,
        ctypes.byref(out)))
    return out


def plan3d(shape, steps, mon_shape=None):
    D, H, W = shape
    Wp = (W + 31) // 32 * 32
    g = _lib.DnGrid(D=D, H=H, W=W, dtype=_lib.DN_F32, pitch_y=Wp, pitch_z=H * Wp, dt=7.0, dl=20.0,
                    axes=_lib.DN_AXES_PHYSICAL, pol=0)
    mon = _lib.DnMonitor(component=_lib.DN_EZ, n_freq=1, box=_lib.box((0, 0, 0), mon_shape or shape))
    out = _lib.DnResidentPlan()
    _lib.check("plan", _lib.lib().dn_fdtd3d_resident_plan(
        ctypes.byref(g), None, ctypes.byref(mon), int(mon_shape is not None), steps, SMS,
        ctypes.byref(out)))
    return out


# a launch of one step does no exchange: bands that store their rows in place would
# overwrite rows that neighbours have not loaded
@pytest.mark.parametrize("adjoint", [False, True])
def test_no_launch_of_a_split_run_is_short(adjoint):
    one = plan2d(256, 256, 40, cells=(256, 256), adjoint=adjoint)
    assert (one.pieces, one.shortest, one.longest) == (1, 40, 40)
    cap = 256  # 256^2 FP32 samples in 64 MB
    for steps in [*range(cap, 4 * cap + 3), 10 * cap + 1, 4001, 100 * cap + 1, 1_000_001]:
        p = plan2d(256, 256, steps, cells=(256, 256), adjoint=adjoint)
        assert p.rows > 0 and p.pieces == -(-steps // cap) and p.longest <= cap
        assert p.shortest >= cap // 2 and p.longest - p.shortest <= 1
    for side in (200, 333, 420, 512, 700):  # down to the fewest steps per launch
        for steps in (60, 65, 97, 129, 1025):
            p = plan2d(side, side, steps, cells=(side, side), adjoint=adjoint)
            assert p.rows == 0 or p.shortest >= 16


def test_no_launch_of_a_split_3d_run_is_short():
    cap = (64 << 20) // (48 ** 3 * 4)
    for steps in [*range(cap, 3 * cap + 3), 50 * cap + 1]:
        p = plan3d((48, 48, 48), steps, (48, 48, 48))
        assert p.rows > 0 and p.pieces == -(-steps // cap) and p.shortest >= cap // 2
    assert plan3d((48, 48, 48), 10_000).pieces == 1


def test_plans_reject_invalid_input():
    out = _lib.DnResidentPlan()
    L = _lib.lib()
    assert L.dn_fdtd2d_resident_plan(None, None, None, 0, 10, 0, SMS, ctypes.byref(out)) == 1
    assert L.dn_fdtd3d_resident_plan(None, None, None, 0, 10, SMS, ctypes.byref(out)) == 1


# one step more than fits, and than fits twice, a launch
@pytest.mark.gpu
@pytest.mark.parametrize("T", [257, 513])
@pytest.mark.parametrize("H,W", [(256, 256), (257, 250)])  # one cluster; the whole chip
def test_a_step_more_than_a_launch_holds(cuda, H, W, T):
    _compare(_engine(H, W, TM, F32, T, [MonitorSpec("all", _lib.DN_EZ, ((0, 1), (0, H), (0, W)),
                                                    [1550.0])]), TM, T)


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(256, 256), (257, 250)])
def test_a_reverse_step_more_than_a_launch_holds(cuda, H, W):
    T = (64 << 20) // (H * W * 4) + 1
    assert plan2d(H, W, T, cells=(H, W), adjoint=True).pieces == 2
    eng = _engine(H, W, TM, F32, T, [MonitorSpec("all", _lib.DN_EZ, ((0, 1), (0, H), (0, W)),
                                                 [1550.0])])
    g = torch.Generator().manual_seed(T)
    lam = torch.randn(6, 1, H, W, dtype=F64, generator=g)
    gm = torch.randn(*eng.accs[0].shape, dtype=F64, generator=g).to(cuda)
    mon_arr = (_lib.DnMonitor * 1)()
    ctypes.memmove(mon_arr, ctypes.byref(eng.mon_arr[0]), ctypes.sizeof(_lib.DnMonitor))
    mon_arr[0].acc = gm.data_ptr()
    buf = eng.curl_buffer(T).zero_()
    buf[0, :, 0, :, :W] = torch.randn(T, H, W, dtype=F64, generator=g).to(cuda, F32)
    rec = eng.curl_record(buf, 0, T)
    got = []
    for ws in (True, False):
        la, lb = torch.zeros_like(eng.A), torch.zeros_like(eng.A)
        la[..., :W] = lam.to(cuda, F32)
        grad = torch.zeros(1, H, eng.Wp, dtype=F64, device=cuda)
        out = _sweep(eng, ws, la, lb, rec, grad, mon_arr, 1, T, T)
        got.append([out[c, ..., :W].clone() for c in _comps(TM)] + [grad[..., :W]])
    for a, b in zip(*got):
        assert rel_l2(a, b) < 2 * _tol(F32, T)


@pytest.mark.gpu
def test_a_3d_step_more_than_a_launch_holds(cuda):
    shape = (48, 48, 48)
    T = (64 << 20) // (48 ** 3 * 4) + 1
    mons = [MonitorSpec("a", _lib.DN_EY, tuple((0, n) for n in shape), (1550.0,))]
    _compare3d(_engine3d(shape, _lib.DN_AXES_PHYSICAL, T, {"pos": [20, 20, 20]}, monitors=mons))


# (shape, rows per warp of a run / of a reverse sweep), FP32 TM: one cluster up to 16
# bands, then the fewest rows for which a band per SM holds the grid
PLANS_F32 = [((1, 1), 1, 1), ((100, 100), 1, 1), ((256, 256), 2, 2), ((257, 256), 1, 1),
             ((300, 413), 1, 1), ((598, 513), 2, 2), ((701, 701), 3, 3), ((1023, 1021), 4, 0),
             ((1200, 1000), 0, 0), ((16, 2048), 2, 2), ((16, 2049), 0, 0)]
PLANS_F64 = [((100, 100), 2, 2), ((333, 270), 1, 1), ((601, 499), 3, 3), ((1100, 450), 4, 0),
             ((598, 513), 0, 0), ((16, 1024), 2, 2), ((16, 1025), 0, 0)]


@pytest.mark.parametrize("dtype,plans", [(F32, PLANS_F32), (F64, PLANS_F64)])
def test_rows_per_warp(dtype, plans):
    for (H, W), run, sweep in plans:
        assert plan2d(H, W, 100, TM, dtype).rows == run
        assert plan2d(H, W, 100, TM, dtype, adjoint=True).rows == sweep
        assert plan2d(H, W, 100, TE, dtype).rows == (run if dtype == F64 else 0)
        assert plan2d(H, W, 100, TE, dtype, adjoint=True).rows == 0
        assert plan2d(H, W, 7, TM, dtype).rows == 0
    assert plan2d(256, 256, 100).cluster and not plan2d(257, 256, 100).cluster


# blocks of three and four rows, the last band and the last block ragged
@pytest.mark.gpu
@pytest.mark.parametrize("H,W,pol,dtype,rows", [
    (701, 701, TM, F32, 3), (1023, 1021, TM, F32, 4), (601, 499, TM, F64, 3), (601, 499, TE, F64, 3),
    (1100, 450, TM, F64, 4), (1099, 449, TE, F64, 4)])
def test_blocks_of_more_rows(cuda, H, W, pol, dtype, rows):
    assert plan2d(H, W, 9, pol, dtype).rows == rows
    for T in (9, 24):
        f = _lib.DN_EZ if pol == TM else _lib.DN_HZ
        _compare(_engine(H, W, pol, dtype, T, [MonitorSpec("box", f, ((0, 1), (H // 2, H // 2 + 5),
                                                                     (3, W - 2)), [1550.0])]), pol, T)


@pytest.mark.gpu
@pytest.mark.parametrize("H,W,dtype", [(701, 701, F32), (601, 499, F64)])
def test_reverse_sweep_of_blocks_of_three_rows(cuda, H, W, dtype):
    assert plan2d(H, W, 9, TM, dtype, adjoint=True).rows == 3
    f = _lib.DN_EZ
    _compare_sweeps(cuda, H, W, dtype, [
        MonitorSpec("row", f, ((0, 1), (H // 2, H // 2 + 1), (0, W)), [1500.0, 1600.0]),
        MonitorSpec("box", f, ((0, 1), (0, (H + 1) // 2), (W // 2, W)), [1550.0])])


# (solves of this size run resident, so the kernel is called by its own entry point)
@pytest.mark.gpu
@pytest.mark.parametrize("pol,comp", [(TM, "Ez"), (TE, "Hz")])
def test_launch_by_launch_kernel_on_a_large_grid_against_the_oracle(cuda, pol, comp):
    n, T = 1024, 30
    g = torch.Generator().manual_seed(n * 1000 + n)
    eps = 1.5 + 2.0 * torch.rand(n, n, dtype=F64, generator=g)  # as _engine makes it
    eng = _engine(n, n, pol, F32, T)
    eng.reset()
    _run(eng, False, 0, T)
    src = {"type": "gaussian_pulse", "row": n // 3, "spread": 300.0, "t0": 700.0}
    o = R.run_2d(eps, dl=20.0, dt=eng.dt, omega=2 * 3.14159 / 1550.0, pml_layers=4,
                 polarization="TM" if pol == TM else "TE", n_steps=T, source=src)
    assert float(o[comp].abs().max()) > 0
    assert rel_l2(eng.field(_lib.COMPONENTS[comp])[0], o[comp]) < 1e-5
