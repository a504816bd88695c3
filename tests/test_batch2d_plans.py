"""How TM batches are dealt to the chip (on the host, for a GPU of 148 multiprocessors),
and the batches that a plan must not break."""

from __future__ import annotations

import ctypes
import os
import subprocess
import sys

import pytest
import torch
from conftest import rel_l2

from diffnano_b200 import _lib
from diffnano_b200.solvers.batch2d import BatchInstance, FDTDBatch2D
from oracle import fdtd_ref as R

SMS = 148
SPIN_LIMIT, POLLS_PER_STEP = 1 << 22, 64


def insts(grids, monitor=False):
    """(H, W, steps) as the C ABI takes them; a plan looks at no address."""
    arr = (_lib.DnBatch2dInst * len(grids))()
    for n, (H, W, T) in enumerate(grids):
        s = arr[n]
        s.H, s.W, s.pitch, s.n_steps, s.dt, s.dl = H, W, (W + 31) // 32 * 32, T, 7.0, 20.0
        s.src_comp = s.mon_comp = _lib.DN_NONE
        s.ce = s.phase = s.acc = 16
        for a in range(2):
            s.b[a] = s.c[a] = 16
            for c in range(3):
                s.f[a][c] = 16
        if monitor:
            s.mon_comp, s.n_freq, s.mon_box = _lib.DN_EZ, 1, _lib.box((0, 0, 0), (1, 1, W))
    cfg = _lib.DnBatch2d(pol=_lib.DN_TM, dtype=_lib.DN_F32, n_inst=len(grids), K=8, tile_rows=16)
    return cfg, arr


def plan(grids, monitor=False, adjoint=False):
    cfg, arr = insts(grids, monitor)
    out = _lib.DnBatch2dPlan()
    _lib.check("plan", _lib.lib().dn_batch2d_resident_plan(ctypes.byref(cfg), arr, int(adjoint), SMS,
                                                           ctypes.byref(out)))
    return out


# a band may wait for a CTA that still runs earlier grids: at most the whole launch
@pytest.mark.parametrize("adjoint", [False, True])
def test_waits_last_as_long_as_the_launch(adjoint):
    p = plan([(100, 100, 900)] * 4, adjoint=adjoint)
    assert p.rows > 0 and p.wait_polls == SPIN_LIMIT + POLLS_PER_STEP * 900
    one = plan([(2368, 64, 8), (8, 8, 8_000_000)], adjoint=adjoint)
    assert one.wait_polls >= SPIN_LIMIT + POLLS_PER_STEP * 8_000_000
    many = plan([(256, 256, 2000)] * 2048, adjoint=adjoint)  # hundreds of grids per CTA
    assert many.wait_polls >= SPIN_LIMIT + POLLS_PER_STEP * 2000 * (2048 * 8 // SMS)
    endless = plan([(100, 100, 2_000_000_000)] * 300, adjoint=adjoint)
    assert endless.wait_polls == 4_000_000_000  # bounded all the same


# the monitors' kernels take a grid per blockIdx.y, which ends at 65535
@pytest.mark.parametrize("n,launches,most", [(65535, 1, 65535), (65536, 2, 65535),
                                             (140_000, 3, 65535)])
def test_a_launch_takes_at_most_65535_grids(n, launches, most):
    p = plan([(16, 32, 8)] * n, monitor=True)
    assert (p.launches, p.most_grids) == (launches, most)


def test_plans_reject_invalid_batches():
    cfg, arr = insts([(100, 100, 900)])
    out = _lib.DnBatch2dPlan()
    call = _lib.lib().dn_batch2d_resident_plan
    assert call(None, arr, 0, SMS, ctypes.byref(out)) == _lib.DN_EINVAL
    arr[0].H = 0
    assert call(ctypes.byref(cfg), arr, 0, SMS, ctypes.byref(out)) == _lib.DN_EINVAL
    cfg.pol, arr[0].H = _lib.DN_TE, 100
    assert call(ctypes.byref(cfg), arr, 0, SMS, ctypes.byref(out)) == _lib.DN_OK and out.rows == 0


NO_MEMORY = """
import ctypes, resource, sys
sys.path.insert(0, sys.argv[1])
from test_batch2d_plans import SMS, _lib, insts
cfg, arr = insts([(16, 32, 8)] * 300_000)
out, call = _lib.DnBatch2dPlan(), _lib.lib().dn_batch2d_resident_plan
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
limit = resource.getrlimit(resource.RLIMIT_AS)
resource.setrlimit(resource.RLIMIT_AS, (used + (1 << 20), limit[1]))
rc = call(ctypes.byref(cfg), arr, 0, SMS, ctypes.byref(out))
resource.setrlimit(resource.RLIMIT_AS, limit)
print(rc, out.rows)
"""


def test_a_host_without_memory_for_a_plan_gets_a_status():
    """(in a process of its own: its address space ends 1 MB further on)"""
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", NO_MEMORY, here], capture_output=True, text=True,
                       timeout=300, cwd=os.path.dirname(here),
                       env={**os.environ, "PYTHONPATH": os.path.dirname(here)})
    assert r.returncode == 0, r.stderr
    assert r.stdout.split() == [str(_lib.DN_ENOMEM), "0"]


def test_a_reverse_sweep_needs_its_arrays():
    size = _lib.lib().dn_batch2d_resident_bytes
    cfg, arr = insts([(100, 100, 900)] * 2)
    assert size(ctypes.byref(cfg), arr, 0) >= 0
    for s in arr:
        s.curl = s.grad = 16
        for a in range(2):
            for c in range(3):
                s.lam[a][c] = 16
    assert size(ctypes.byref(cfg), arr, 1) >= 0
    arr[1].curl = None
    assert size(ctypes.byref(cfg), arr, 1) == -1
    arr[1].curl, arr[1].grad = 16, None
    assert size(ctypes.byref(cfg), arr, 1) == -1
    arr[1].grad, arr[1].lam[1][2] = 16, None
    assert size(ctypes.byref(cfg), arr, 1) == -1
    arr[0].H = 0
    assert size(ctypes.byref(cfg), arr, 0) == -1


def _rows(specs, dtype, curl=False, adjoint=False):
    cfg, arr = insts([(*s.grid_shape, s.n_steps) for s in specs])
    cfg.dtype = _lib.DN_F32 if dtype == torch.float32 else _lib.DN_F64
    for s in arr:
        s.curl = 16 if curl else None
    out = _lib.DnBatch2dPlan()
    _lib.check("plan", _lib.lib().dn_batch2d_resident_plan(ctypes.byref(cfg), arr, int(adjoint), SMS,
                                                           ctypes.byref(out)))
    return out.rows


# the two batches of tests/test_batch2d_resident.py run with 1 and 4 rows per warp and
# sweep with 1 and 2; here the runs with two rows
@pytest.mark.gpu
@pytest.mark.parametrize("shapes,dtype", [([(300, 413)] * 3, torch.float32),
                                          ([(300, 400), (200, 129)], torch.float64)])
def test_a_batch_with_two_rows_per_warp(cuda, shapes, dtype):
    specs = [BatchInstance(grid_shape=s, n_steps=24 + 6 * (s[0] < 300), pml_layers=4,
                           source={"type": "gaussian_pulse", "row": 20, "spread": 100.0, "t0": 80.0})
             for s in shapes]
    assert _rows(specs, dtype) == 2
    g = torch.Generator().manual_seed(7)
    eps = [(1.5 + 2.0 * torch.rand(*s, dtype=torch.float64, generator=g)).to(cuda) for s in shapes]
    fields, _ = FDTDBatch2D(specs, "TM", dtype, cuda, tile_rows=16).forward(eps)
    for spec, e, f in zip(specs, eps, fields):
        o = R.run_2d(e.cpu(), dl=spec.dl, dt=spec.dt, omega=spec.omega, pml_layers=4,
                     n_steps=spec.n_steps, source=spec.source)
        assert rel_l2(f, o["Ez"]) < (1e-5 if dtype == torch.float32 else 1e-12)


@pytest.mark.gpu
def test_a_recorded_run_needs_curl_records(cuda):
    """A plan of grids without curl arrays refuses to record, and one of another type to
    run (nothing is launched)."""
    L = _lib.lib()
    cfg, arr = insts([(64, 64, 20)] * 2)
    n, ws = int(L.dn_batch2d_resident_bytes(ctypes.byref(cfg), arr, 0)), ctypes.c_int64(0)
    assert n > 0
    host = (ctypes.c_ubyte * n)()
    _lib.check("pack", L.dn_batch2d_resident_pack(ctypes.byref(cfg), arr, 0, host, n,
                                                  ctypes.byref(ws)))
    run = L.dn_batch2d_run_resident
    assert run(ctypes.byref(cfg), 16, host, 16, 16, 1 << 40, 1, None, None) == _lib.DN_EINVAL
    cfg.dtype = _lib.DN_F64
    assert run(ctypes.byref(cfg), 16, host, 16, 16, 1 << 40, 0, None, None) == _lib.DN_EINVAL


@pytest.mark.gpu
def test_a_band_waits_out_a_long_run_on_its_neighbours_cta(cuda):
    """One tiny grid of millions of steps on a CTA that a grid of a band per SM needs
    too: its other bands wait for seconds."""
    src = {"type": "gaussian_pulse", "row": 3, "spread": 100.0, "t0": 20.0}
    long = BatchInstance(grid_shape=(8, 8), n_steps=8_000_000, pml_layers=2, source=src)
    wide = BatchInstance(grid_shape=(16 * SMS, 64), n_steps=8, pml_layers=4,
                         source={**src, "row": 16 * SMS // 2})
    g = torch.Generator().manual_seed(2)
    eps = [(1.5 + 2.0 * torch.rand(*s.grid_shape, dtype=torch.float64, generator=g)).to(cuda)
           for s in (long, wide)]
    b = FDTDBatch2D([long, wide], "TM", torch.float32, cuda, tile_rows=16)
    fields, _ = b.forward(eps)
    assert b.uses_resident(True, False)
    alone, _ = FDTDBatch2D([wide], "TM", torch.float32, cuda, tile_rows=16).forward(eps[1:])
    assert rel_l2(fields[1], alone[0]) < 1e-6 and float(alone[0].abs().max()) > 0
