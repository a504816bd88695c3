"""Resident 2-D runs (all steps in one launch, fields in registers) against the
launch-by-launch kernels, through the C ABI: with a workspace dn_fdtd2d_run_ws
takes the resident path, dn_fdtd2d_run steps launch by launch.

Both do the same update with different groupings of the constant factors, so a
step differs by a few roundings and a run of T steps by at most about 2 T units
of round-off (relative L2; measured ~10x below).
"""

from __future__ import annotations

import ctypes

import pytest
import torch
from conftest import rel_l2

from diffnano_b200 import _lib
from diffnano_b200.solvers import _setup
from diffnano_b200.solvers._engine import Engine, MonitorSpec

EPS = {torch.float32: 2.0 ** -24, torch.float64: 2.0 ** -53}


def _tol(dtype, T):
    return 2 * T * EPS[dtype]


def _engine(H, W, pol, dtype, T, monitors=(), probe=None, src=True):
    dl, dt = 20.0, 0.5 * 20.0 / 2 ** 0.5
    inj = _lib.DN_EZ if pol == _lib.DN_TM else _lib.DN_HZ
    s = {"type": "gaussian_pulse", "row": H // 3, "spread": 300.0, "t0": 700.0}
    eng = Engine(is3d=False, shape=(H, W), dl=dl, dt=dt, pml_layers=min(4, H // 2, W // 2),
                 dtype=dtype, device=torch.device("cuda", 0), n_steps=T,
                 wave=_setup.waveform_table(T, dt, 2 * 3.14159 / 1550.0, s),
                 src_box=_setup.source_box_2d((H, W), s) if src else None,
                 src_comp=inj if src else _lib.DN_NONE, monitors=monitors, probe=probe, pol=pol)
    g = torch.Generator().manual_seed(H * 1000 + W)
    eng.set_eps(1.5 + 2.0 * torch.rand(H, W, dtype=torch.float64, generator=g))
    eng.state0 = torch.randn(6, 1, H, W, dtype=torch.float64, generator=g)
    return eng


def _start(eng):
    eng.reset()
    eng.A[..., : eng.shape3[2]] = eng.state0.to(eng.device, eng.dtype)


def _comps(pol):
    return ((_lib.DN_EZ, _lib.DN_HX, _lib.DN_HY) if pol == _lib.DN_TM
            else (_lib.DN_HZ, _lib.DN_EX, _lib.DN_EY))


def _run(eng, resident, t0, T, rec=None):
    """State and monitor sums after T steps; the resident path or the other."""
    if resident:
        assert int(_lib.lib().dn_fdtd2d_workspace_bytes(
            ctypes.byref(eng.grid), ctypes.byref(eng.src), eng.mon_arr, len(eng.monitors),
            eng.n_steps)) >= 0
        eng.run(t0, T, record=rec)
    else:
        out = ctypes.c_int32(0)
        fa, fb = (eng.B, eng.A) if eng.cur_b else (eng.A, eng.B)
        rc = _lib.lib().dn_fdtd2d_run(
            ctypes.byref(eng.grid), eng._ptrs(fa), eng._ptrs(fb), eng.ce.data_ptr(),
            ctypes.byref(eng.cpml), ctypes.byref(eng.src), eng.mon_arr, len(eng.monitors),
            ctypes.byref(eng.probe), ctypes.byref(rec) if rec is not None else None, t0, T,
            eng.status.data_ptr(),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(out))
        _lib.check("dn_fdtd2d_run", rc)
        eng.cur_b ^= bool(out.value)
    eng.check_status()


def _compare(eng, pol, T, t0=0):
    got = []
    for resident in (True, False):
        _start(eng)
        _run(eng, resident, t0, T)
        got.append(([eng.field(c).clone() for c in _comps(pol)], [a.clone() for a in eng.accs],
                    None if eng.probe_out is None else eng.probe_out.clone()))
    tol = _tol(eng.dtype, T)
    for a, b in zip(*[g[0] for g in got]):
        assert rel_l2(a, b) < tol
    for a, b in zip(*[g[1] for g in got]):
        assert rel_l2(a, b) < 4 * tol
    if got[0][2] is not None:
        assert rel_l2(got[0][2], got[1][2]) < 4 * tol


# FP32 TE runs stay launch by launch
KINDS = [(_lib.DN_TM, torch.float32), (_lib.DN_TM, torch.float64), (_lib.DN_TE, torch.float64)]

# edges of lanes (4 / 2 columns), strips (128 / 64), blocks of 1 .. 4 rows and
# bands; one band, a cluster of bands, bands over the whole chip
SHAPES = [(1, 1), (2, 3), (5, 130), (16, 128), (17, 127), (100, 100), (129, 129), (256, 255),
          (300, 413), (333, 270), (598, 513), (1024, 1022)]


@pytest.mark.gpu
@pytest.mark.parametrize("pol,dtype", KINDS)
@pytest.mark.parametrize("H,W", SHAPES)
def test_fields_from_a_random_state(cuda, H, W, pol, dtype):
    for T in (9, 24):  # odd and even: the result ends in either set
        _compare(_engine(H, W, pol, dtype, T), pol, T)


@pytest.mark.gpu
@pytest.mark.parametrize("pol,dtype", KINDS)
def test_monitors_and_probe(cuda, pol, dtype):
    """Row, column, ragged box and one-cell monitors on all three fields, with
    aligned and unaligned columns, a probe, and a start after step 0."""
    H, W, T = 97, 141, 40
    f, a, b = _comps(pol)
    mons = [MonitorSpec("row", f, ((0, 1), (60, 61), (0, W)), [1500.0, 1550.0, 1600.0]),
            MonitorSpec("col", a, ((0, 1), (0, H), (7, 8)), [1550.0]),
            MonitorSpec("box", b, ((0, 1), (3, 50), (126, 135)), [1400.0 + 40 * k for k in range(6)]),
            MonitorSpec("quad", f, ((0, 1), (90, 97), (120, 132)), [1550.0])]
    eng = _engine(H, W, pol, dtype, T, mons, probe=(f, (0, 33, 131)))
    _compare(eng, pol, T - 3, t0=3)


@pytest.mark.gpu
def test_samples_in_pieces(cuda):
    """A whole-grid monitor whose samples exceed the workspace's share: the run
    goes in pieces, each with its own DFT."""
    H, W, T = 256, 256, 300
    mons = [MonitorSpec("all", _lib.DN_EZ, ((0, 1), (0, H), (0, W)), [1550.0])]
    _compare(_engine(H, W, _lib.DN_TM, torch.float32, T, mons), _lib.DN_TM, T)


@pytest.mark.gpu
@pytest.mark.parametrize("pol,dtype", KINDS)
@pytest.mark.parametrize("H,W", [(40, 45), (300, 413)])
def test_curl_record(cuda, H, W, pol, dtype):
    T = 20
    eng = _engine(H, W, pol, dtype, T)
    recs = []
    for resident in (True, False):
        _start(eng)
        buf = eng.curl_buffer(T).zero_()
        _run(eng, resident, 2, T - 4, eng.curl_record(buf, 1, T - 1))
        recs.append(buf[..., :W].clone())
    assert rel_l2(recs[0], recs[1]) < 4 * _tol(dtype, T)
    assert not recs[0][:, 0].any() and recs[0][:, 1:17].any()


def test_workspace_bytes_reject_invalid_input():
    L = _lib.lib()
    g = _lib.DnGrid(D=1, H=32, W=32, dtype=_lib.DN_F32, pitch_y=32, pitch_z=1024, dt=7.0, dl=20.0,
                    axes=0, pol=_lib.DN_TM)
    assert L.dn_fdtd2d_workspace_bytes(None, None, None, 0, 10) == -1
    assert L.dn_fdtd2d_workspace_bytes(ctypes.byref(g), None, None, 1, 10) == -1
    g.H = 0
    assert L.dn_fdtd2d_workspace_bytes(ctypes.byref(g), None, None, 0, 10) == -1


def _sweep(eng, ws, la, lb, rec, grad, mon_arr, n_mon, t_end, T):
    L, out = _lib.lib(), ctypes.c_int32(0)
    args = (ctypes.byref(eng.grid), eng._ptrs(la), eng._ptrs(lb), eng.ce.data_ptr(),
            ctypes.byref(eng.cpml), ctypes.byref(rec), grad.data_ptr(), mon_arr, n_mon, t_end, T,
            eng.status.data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
            ctypes.byref(out))
    if ws:
        _lib.check("ws", L.dn_fdtd2d_adjoint_ws(*args, *eng._workspace()))
    else:
        _lib.check("steps", L.dn_fdtd2d_adjoint(*args))
    eng.check_status(extra=(grad,))
    return lb if out.value else la


def _compare_sweeps(cuda, H, W, dtype, mons):
    """From random adjoint fields, curl terms and a running gradient, with monitors
    whose gradients enter before every step."""
    for T in (9, 24):
        eng = _engine(H, W, _lib.DN_TM, dtype, T + 3, mons)
        g = torch.Generator().manual_seed(T)
        rand = lambda *s: torch.randn(*s, dtype=torch.float64, generator=g)  # noqa: E731
        lam, curl, grad0 = rand(6, 1, H, W), rand(T, H, W), rand(1, H, W)
        gm = [rand(*a.shape).to(cuda) for a in eng.accs]
        mon_arr = (_lib.DnMonitor * len(mons))()
        for m in range(len(mons)):
            ctypes.memmove(ctypes.byref(mon_arr[m]), ctypes.byref(eng.mon_arr[m]),
                           ctypes.sizeof(_lib.DnMonitor))
            mon_arr[m].acc = gm[m].data_ptr()
        buf = eng.curl_buffer(T).zero_()
        buf[0, :, 0, :, :W] = curl.to(cuda, dtype)
        rec = eng.curl_record(buf, 2, T)
        got = []
        for ws in (True, False):
            la, lb = torch.zeros_like(eng.A), torch.zeros_like(eng.A)
            la[..., :W] = lam.to(cuda, dtype)
            grad = torch.zeros(1, H, eng.Wp, dtype=torch.float64, device=cuda)
            grad[..., :W] = grad0.to(cuda)
            out = _sweep(eng, ws, la, lb, rec, grad, mon_arr, len(mons), T + 2, T)
            got.append([out[c, ..., :W].clone() for c in _comps(_lib.DN_TM)] + [grad[..., :W]])
        for a, b in zip(*got):
            assert rel_l2(a, b) < 2 * _tol(dtype, T)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("H,W", [s for s in SHAPES if s[0] * s[1] < 500_000])
def test_reverse_sweep(cuda, H, W, dtype):
    f = _lib.DN_EZ
    _compare_sweeps(cuda, H, W, dtype, [
        MonitorSpec("row", f, ((0, 1), (H // 2, H // 2 + 1), (0, W)), [1500.0, 1600.0]),
        MonitorSpec("box", f, ((0, 1), (0, (H + 1) // 2), (W // 2, W)), [1550.0])])


# what a block reads a step ahead and what it does not: rows that end inside a lane's
# columns, rows of a wider table, two of a block's rows, columns off the 16 bytes; two
# monitors on the same cells, the one read ahead first or second
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("boxes", [[((50, 51), (8, 61))], [((40, 45), (4, 132))],
                                   [((40, 45), (4, 131))], [((70, 71), (3, 140))],
                                   [((60, 61), (0, 141)), ((58, 63), (2, 99))],
                                   [((58, 63), (2, 99)), ((60, 61), (0, 141))],
                                   [((96, 97), (136, 141)), ((96, 97), (136, 141))]])
@pytest.mark.parametrize("H", [97, 390])
def test_reverse_sweep_monitors(cuda, H, boxes, dtype):
    _compare_sweeps(cuda, H, 141, dtype, [
        MonitorSpec(str(n), _lib.DN_EZ, ((0, 1), *b), [1550.0]) for n, b in enumerate(boxes)])
