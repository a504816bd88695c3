"""Single 2-D solves that do not run resident (FP32 TE, a few steps) take one cluster
launch where the grid fits a thread-block cluster and its warps have little to walk."""

from __future__ import annotations

import pytest
import test_resident_plans as plans
import torch
from conftest import rel_l2
from test_batch2d_kernels import _Recorder

import diffnano_b200 as dn
from diffnano_b200 import _lib
from diffnano_b200.solvers.batch2d import BatchInstance, fits_cluster
from oracle import fdtd_ref as R

F32, F64 = torch.float32, torch.float64


def test_what_fits_a_cluster():
    def fits(H, W, pol="TE", dtype=F32, T=10, mon=None):
        return fits_cluster(BatchInstance(grid_shape=(H, W), n_steps=T, monitor=mon), pol, dtype)

    assert fits(256, 256) and fits(40, 2100, "TM") and fits(256, 256, "TM", F64)
    assert not fits(1024, 1024) and not fits(700, 700, "TM", F64) and not fits(64, 64, T=0)
    assert fits(64, 64, mon={"row": 3, "wavelengths_nm": [1550.0]})
    assert not fits(64, 64, mon={"row": 3, "wavelengths_nm": []})


def test_no_other_grid_is_one_for_the_cluster():
    """What FDTDSolver2D takes for granted: beside FP32 TE and runs of under 8 steps, no
    grid within the cluster rule's 24 pieces lacks a resident plan."""
    for pol, dtype in ((plans.TM, F32), (plans.TM, F64), (plans.TE, F64)):
        assert plans.plan2d(100, 100, 8, pol, dtype).rows > 0
        assert plans.plan2d(100, 100, 7, pol, dtype).rows == 0
        for pieces in range(1, 25):
            for turns in range(1, 24 // pieces + 1):
                H, W = 256 * turns, 32 * pieces
                assert plans.plan2d(H, W, 8, pol, dtype).rows > 0


def _forward(monkeypatch, solver, *a, **kw):
    with monkeypatch.context() as m:
        rec = _Recorder(_lib.lib())
        m.setattr(_lib, "lib", lambda: rec)
        return rec, solver.forward(*a, **kw)


@pytest.mark.parametrize("shape,pol,dtype,T,want", [
    ((100, 100), "TM", F32, 37, True), ((100, 100), "TM", F32, 38, False),
    ((256, 256), "TM", F64, 25, True), ((256, 256), "TM", F64, 26, False),
    ((16, 32), "TM", F32, 60, True), ((16, 32), "TM", F32, 61, False),
    ((256, 768), "TM", F32, 10, True), ((256, 769), "TM", F32, 11, False),
    ((256, 768), "TE", F32, 500, True), ((257, 513), "TE", F32, 500, False),
    ((257, 513), "TE", F32, 7, True), ((256, 256), "TE", F64, 500, False)])
def test_which_solves_are_for_the_cluster(shape, pol, dtype, T, want):
    s = dn.FDTDSolver2D(grid_shape=shape, polarization=pol, n_steps=T, dtype=dtype)
    assert s._for_cluster(None) == s._for_cluster([{"row": 3}]) == want
    assert not s._for_cluster([{"row": 3}, {"row": 4}])
    assert not s._for_cluster(m for m in [{"row": 3}])  # (not looked into)


# (shape, polarisation, type, steps): FP32 TE, a row of 24 pieces, a few steps
CASES = [((100, 100), "TE", F32, 60), ((131, 77), "TE", F32, 60), ((20, 768), "TE", F32, 60),
         ((100, 100), "TM", F32, 5), ((100, 100), "TE", F64, 7), ((129, 131), "TM", F32, 33), ((129, 131), "TM", F64, 20),
         ((20, 1128), "TM", F32, 3)]


@pytest.mark.gpu
@pytest.mark.parametrize("shape,pol,dtype,T", CASES)
@pytest.mark.parametrize("monitors", [0, 1])
def test_cluster_solve(cuda, monkeypatch, shape, pol, dtype, T, monitors):
    H, W = shape
    src = {"type": "gaussian_pulse", "row": 6, "spread": 100.0, "t0": 150.0}
    mon = {"row": 10, "wavelengths_nm": [1500.0, 1600.0]}
    s = dn.FDTDSolver2D(grid_shape=shape, polarization=pol, pml_layers=4, n_steps=T, device=cuda,
                        dtype=dtype, monitors=[mon] if monitors else None)
    g = torch.Generator().manual_seed(H)
    tol = 1e-5 if dtype == F32 else 1e-12
    for _ in range(2):  # the second solve reuses what the first one made
        eps = 1.5 + 2.0 * torch.rand(*shape, dtype=F64, generator=g)
        rec, r = _forward(monkeypatch, s, eps.to(cuda), source=dict(src))
        assert rec.ran == ["dn_batch2d_forward_cluster"]
        first = "Ez" if pol == "TM" else "Hz"
        o = R.run_2d(eps, dl=s.dl, dt=s.dt, omega=s.omega, pml_layers=4, polarization=pol,
                     n_steps=T, source=src, monitors=[{"component": first, "box": ((10, 11), (0, W)),
                                                       "wavelengths_nm": mon["wavelengths_nm"]}])
        assert rel_l2(r.field[0], o[first]) < tol
        if monitors:
            d = torch.view_as_real(r.metadata["monitors"][0]["dft"])
            assert rel_l2(d.reshape(o["monitors"][0].shape), o["monitors"][0]) < tol
    assert len(s._cluster_cache) == 1


@pytest.mark.gpu
def test_other_solves_keep_their_path(cuda, monkeypatch):
    eps = torch.full((100, 100), 2.0, dtype=F64, device=cuda)
    src = {"type": "gaussian_pulse", "row": 6}
    two = [{"row": 10}, {"col": 10}]
    other = [{"component": "Ex", "row": 10}]
    for pol, kw, probe in (("TM", {}, None), ("TE", {}, [3, 4]), ("TE", {"monitors": two}, None),
                           ("TE", {"monitors": other}, None), ("TE", {"grid_shape": (20, 769)}, None),
                           ("TM", {"grid_shape": (40, 2100)}, None)):
        s = dn.FDTDSolver2D(polarization=pol, n_steps=60, device=cuda, **kw)
        e = eps.new_full(s.grid_shape, 2.0)
        rec, r = _forward(monkeypatch, s, e, source={**src, **({"probe": probe} if probe else {})})
        assert rec.ran == [] and len(s._engine_cache) == 1
    e = eps.clone().requires_grad_(True)
    rec, r = _forward(monkeypatch, dn.FDTDSolver2D(polarization="TE", n_steps=60, device=cuda), e,
                      source=src)
    assert rec.ran == [] and r.field.requires_grad
