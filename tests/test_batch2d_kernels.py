"""Which kernel a batched solve launches, and TM batches on the kernels that they use
without a resident plan (no room for its workspace, or a grid that does not fit)
against the CPU FP64 oracle."""

from __future__ import annotations

from dataclasses import replace

import pytest
import torch
from conftest import rel_l2

from diffnano_b200 import _lib
from diffnano_b200.solvers import batch2d
from diffnano_b200.solvers.batch2d import BatchInstance, FDTDBatch2D
from oracle import fdtd_ref as R

SHAPES, STEPS = [(40, 36), (70, 130), (33, 90)], [60, 45, 90]


def _specs():
    return [BatchInstance(grid_shape=s, n_steps=T, dl=20.0, wavelength_nm=1550.0, pml_layers=4,
                          courant=0.5, source={"type": "gaussian_pulse", "row": 6, "spread": 300.0,
                                               "t0": 300.0},
                          monitor={"row": 12, "wavelengths_nm": [1500.0, 1600.0]})
            for s, T in zip(SHAPES, STEPS)]


def _eps():
    g = torch.Generator().manual_seed(11)
    return [1.5 + 2.0 * torch.rand(*s, dtype=torch.float64, generator=g) for s in SHAPES]


class _Recorder:
    """The library, with the names of the batch entry points that run kernels."""

    def __init__(self, lib):
        self.lib, self.ran = lib, []

    def __getattr__(self, name):
        if name in ("dn_batch2d_forward", "dn_batch2d_forward_cluster", "dn_batch2d_run_resident",
                    "dn_batch2d_backward"):
            self.ran.append(name)
        return getattr(self.lib, name)


def _forward(monkeypatch, batch, eps):
    with monkeypatch.context() as m:
        rec = _Recorder(_lib.lib())
        m.setattr(_lib, "lib", lambda: rec)
        fields, dfts = batch.forward(eps)
    return rec.ran[-1], fields, dfts


def test_an_explicit_cluster_comes_before_a_resident_plan():
    b = FDTDBatch2D.__new__(FDTDBatch2D)
    b._plans, b._record = {False: None, True: None}, True
    for cluster in (None, False, True):
        b.cluster = cluster
        assert b.uses_resident(True, False) == (cluster is not True)
        assert b.uses_resident(True, True) and b.uses_resident(False, True)


# at most 90 steps of a few roundings each: 1e-5 is 2 T units of 2^-24
@pytest.mark.gpu
@pytest.mark.parametrize("dtype,tol", [(torch.float32, 1e-5), (torch.float64, 1e-12)])
@pytest.mark.parametrize("cluster,plan,kernel", [
    (None, True, "dn_batch2d_run_resident"), (False, True, "dn_batch2d_run_resident"),
    (True, True, "dn_batch2d_forward_cluster"), (None, False, "dn_batch2d_forward_cluster"),
    (False, False, "dn_batch2d_forward")])
def test_tm_kernels_against_the_oracle(cuda, monkeypatch, cluster, plan, kernel, dtype, tol):
    specs, eps = _specs(), _eps()
    if not plan:
        monkeypatch.setattr(FDTDBatch2D, "_plan_resident", lambda self: None)
    rows = [8, 16, 32] if kernel == "dn_batch2d_forward" else [16]
    for tile_rows in rows:
        b = FDTDBatch2D(specs, "TM", dtype, cuda, tile_rows=tile_rows, cluster=cluster)
        ran, fields, dfts = _forward(monkeypatch, b, [e.to(cuda) for e in eps])
        assert ran == kernel
        for spec, e, f, d in zip(specs, eps, fields, dfts):
            o = R.run_2d(e, dl=spec.dl, dt=spec.dt, omega=spec.omega,
                         pml_layers=4, n_steps=spec.n_steps, source=spec.source,
                         monitors=[{"component": "Ez", "box": ((12, 13), (0, spec.grid_shape[1])),
                                    "wavelengths_nm": spec.monitor["wavelengths_nm"]}])
            assert rel_l2(f, o["Ez"]) < tol
            got = torch.view_as_real(d.to(torch.complex128)).reshape(o["monitors"][0].shape)
            assert rel_l2(got, o["monitors"][0]) < tol


@pytest.mark.gpu
def test_a_graph_replay_keeps_the_cluster_kernel(cuda, monkeypatch):
    eps = [e.to(cuda) for e in _eps()]
    b = FDTDBatch2D(_specs(), "TM", torch.float32, cuda, tile_rows=16, cluster=True)
    ran, fields, _ = _forward(monkeypatch, b, eps)
    replayed, _ = b.forward_graphed(eps)
    assert ran == "dn_batch2d_forward_cluster"
    assert all(torch.equal(x, y) for x, y in zip(fields, replayed))


@pytest.mark.gpu
def test_tile_heights_are_timed_once(cuda, monkeypatch):
    """A batch that alternates between solves with and without gradient keeps the tile
    height it has chosen."""
    calls = []
    monkeypatch.setattr(batch2d, "autotune_tile_rows", lambda b: calls.append(1) or 32)
    eps = [e.to(cuda) for e in _eps()]
    b = FDTDBatch2D([replace(s, monitor=None) for s in _specs()], "TE", torch.float64, cuda)
    for _ in range(2):
        b.forward(eps)
        fields, _ = b.forward([e.requires_grad_(True) for e in eps])
        torch.autograd.grad(sum(f.sum() for f in fields), eps)
        eps = [e.detach() for e in eps]
    assert len(calls) == 1 and b.tile_rows == 32
