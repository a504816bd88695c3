"""Batched TM grids held on the chip (``dn_batch2d_run_resident``) against
single-grid solves and the persistent kernel: ragged instances, more bands than
SMs, several launches for one batch, and gradients from recorded curl terms."""

from __future__ import annotations

import pytest
import torch
from conftest import rel_l2

import diffnano_b200 as dn
from diffnano_b200.solvers.batch2d import BatchInstance, FDTDBatch2D

pytestmark = pytest.mark.gpu


def _spec(H, W, T, mon):
    src = {"type": "gaussian_pulse", "row": H // 4, "spread": 300.0, "t0": 900.0}
    return BatchInstance(grid_shape=(H, W), n_steps=T, dl=20.0, wavelength_nm=1550.0,
                         pml_layers=4, courant=0.5, source=src, monitor=mon)


def _eps(specs, cuda, seed):
    g = torch.Generator().manual_seed(seed)
    return [(1.5 + 2.0 * torch.rand(*s.grid_shape, dtype=torch.float64, generator=g)).to(cuda)
            for s in specs]


def _single(spec, dtype, cuda, eps):
    s = dn.FDTDSolver2D(grid_shape=spec.grid_shape, dl=spec.dl, wavelength_nm=spec.wavelength_nm,
                        pml_layers=spec.pml_layers, n_steps=spec.n_steps, courant=spec.courant,
                        device=cuda, dtype=dtype, use_checkpoint=True, checkpoint_segments=4,
                        monitors=[spec.monitor] if spec.monitor else None)
    return s.forward(eps, source=dict(spec.source))


ROW = {"row": 30, "wavelengths_nm": [1500.0, 1550.0, 1600.0]}
BOX = {"box": [[3, 31], [5, 34]], "wavelengths_nm": [1550.0]}
# few grids (one row per warp), ragged; and more bands than SMs (longer lists)
FEW = [_spec(40, 45, 60, ROW), _spec(129, 130, 33, BOX), _spec(64, 513, 90, None),
       _spec(33, 36, 8, ROW)]
MANY = [_spec(60 + 17 * (b % 9), 50 + 61 * (b % 7), 24 + 5 * (b % 5), ROW if b % 3 else BOX)
        for b in range(60)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("specs", [FEW, MANY], ids=["few", "many"])
def test_fields_and_dfts_match_single_grids(cuda, specs, dtype):
    eps = _eps(specs, cuda, 1)
    b = FDTDBatch2D(specs, "TM", dtype, cuda)
    fields, dfts = b.forward(eps)
    assert b.uses_resident(True, False)
    tol = 1e-6 if dtype == torch.float32 else 1e-13
    for spec, e, f, d in zip(specs, eps, fields, dfts):
        r = _single(spec, dtype, cuda, e)
        assert rel_l2(f, r.field[0]) < tol
        if spec.monitor:
            dr = r.metadata["monitors"][0]["dft"]
            assert rel_l2(torch.view_as_real(d), torch.view_as_real(dr)) < tol


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("specs", [FEW, MANY], ids=["few", "many"])
def test_gradients_match_the_checkpoint_path(cuda, specs, dtype):
    g = torch.Generator().manual_seed(2)
    w = [torch.randn(*s.grid_shape, dtype=torch.float64, generator=g).to(cuda) for s in specs]
    out = []
    for kw in ({}, {"checkpoint_interval": 7, "tile_rows": 16}):
        eps = [e.requires_grad_(True) for e in _eps(specs, cuda, 3)]
        b = FDTDBatch2D(specs, "TM", dtype, cuda, **kw)
        fields, dfts = b.forward(eps)
        assert b.uses_resident(False, True) == (not kw)
        loss = sum((f.double() * x).sum() for f, x in zip(fields, w))
        loss = loss + sum((d.abs() ** 2).sum() for d in dfts if d is not None)
        out.append(torch.autograd.grad(loss, eps))
        if not kw:  # the batch keeps its record: a second call gives the same bits
            fields, dfts = b.forward(eps)
            loss = sum((f.double() * x).sum() for f, x in zip(fields, w))
            loss = loss + sum((d.abs() ** 2).sum() for d in dfts if d is not None)
            assert all(torch.equal(x, y) for x, y in zip(out[0], torch.autograd.grad(loss, eps)))
    tol = 1e-5 if dtype == torch.float32 else 1e-12
    for a, c in zip(*out):
        assert rel_l2(a, c) < tol


def test_several_launches_for_one_batch(cuda):
    """Samples beyond one launch's share: the grids go in groups, each result the
    one of a batch of its own."""
    mon = {"box": [[0, 128], [0, 128]], "wavelengths_nm": [1550.0]}
    specs = [_spec(128, 128, 2000 - 100 * b, mon) for b in range(6)]
    eps = _eps(specs, cuda, 5)
    fields, dfts = FDTDBatch2D(specs, "TM", torch.float64, cuda).forward(eps)
    for n in (0, 3, 5):
        f1, d1 = FDTDBatch2D(specs[n:n + 1], "TM", torch.float64, cuda).forward(eps[n:n + 1])
        assert rel_l2(fields[n], f1[0]) < 1e-13
        assert rel_l2(torch.view_as_real(dfts[n]), torch.view_as_real(d1[0])) < 1e-13


def test_graph_replays_the_resident_gradient(cuda):
    specs = FEW[:2] + FEW[3:]
    eps_a, eps_b = _eps(specs, cuda, 6), _eps(specs, cuda, 7)
    b = FDTDBatch2D(specs, "TM", torch.float32, cuda)
    fom, grads = b.fom_gradient_graphed(eps_a)
    first = fom.clone(), [x.clone() for x in grads]
    b.fom_gradient_graphed(eps_b)
    fom, grads = b.fom_gradient_graphed(eps_a)
    assert b.uses_resident(False, True)
    assert torch.equal(fom, first[0]) and all(torch.equal(x, y) for x, y in zip(grads, first[1]))
    e = [x.clone().requires_grad_(True) for x in eps_a]
    _, dfts = FDTDBatch2D(specs, "TM", torch.float32, cuda).forward(e)
    want = torch.autograd.grad(sum((d.abs() ** 2).sum() for d in dfts), e)
    for x, y in zip(grads, want):
        assert rel_l2(x, y) < 1e-12
