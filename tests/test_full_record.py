"""Gradients from the curl terms recorded during the forward run (the default
where they fit) against those from checkpoints and replay, and the way back to
checkpoints when the record cannot be allocated."""

from __future__ import annotations

import pytest
import torch

import diffnano_b200 as dn
from diffnano_b200.solvers import fom_abs2
from diffnano_b200.solvers._engine import Engine

pytestmark = pytest.mark.gpu


def _gradient(solver, eps, src):
    e = eps.clone().requires_grad_(True)
    r = solver.forward(e, source=dict(src))
    fom = fom_abs2(r.metadata["monitors"][0]["dft"]) + (r.field.double() ** 2).sum()
    (g,) = torch.autograd.grad(fom, e)
    return r.field.detach(), g


def _solver3d(cuda, **kw):
    mon = [{"component": "Ex", "plane": "xy", "z": 16, "wavelengths_nm": [1550.0]}]
    return dn.FDTDSolver3D(grid_shape=(24, 20, 36), pml_layers=4, n_steps=37, device=cuda,
                           cpml_axes="physical", monitors=mon, **kw)


def test_record_equals_checkpoints_bit_for_bit(cuda):
    g = torch.Generator().manual_seed(3)
    eps = (1.5 + 2.0 * torch.rand(24, 20, 36, dtype=torch.float64, generator=g)).to(cuda)
    src = {"type": "gaussian_pulse", "plane": "xy", "z": 7, "component": "Ex"}
    f0, g0 = _gradient(_solver3d(cuda), eps, src)
    f1, g1 = _gradient(_solver3d(cuda, use_checkpoint=True, checkpoint_segments=3), eps, src)
    assert torch.equal(f0, f1) and torch.equal(g0, g1) and g0.abs().max() > 0


def test_checkpoints_when_the_record_does_not_fit(cuda, monkeypatch):
    g = torch.Generator().manual_seed(4)
    eps = (1.5 + 2.0 * torch.rand(24, 20, 36, dtype=torch.float64, generator=g)).to(cuda)
    src = {"type": "gaussian_pulse", "plane": "xy", "z": 7, "component": "Ex"}
    f0, g0 = _gradient(_solver3d(cuda), eps, src)
    real, asked = Engine.curl_buffer, []

    def small(self, n):
        asked.append(n)
        if n == 37:
            raise torch.OutOfMemoryError("no room for the record")
        return real(self, n)

    monkeypatch.setattr(Engine, "curl_buffer", small)
    f1, g1 = _gradient(_solver3d(cuda), eps, src)
    assert asked[0] == 37 and 0 < asked[1] < 37
    assert torch.equal(f0, f1) and torch.equal(g0, g1)


@pytest.mark.parametrize("make", [
    lambda dev: dn.FDTDSolver2D(grid_shape=(20, 30), pml_layers=4, n_steps=0, device=dev),
    lambda dev: dn.FDTDSolver2D(grid_shape=(20, 30), polarization="TE", n_steps=0, device=dev),
    lambda dev: dn.FDTDSolver3D(grid_shape=(8, 9, 10), pml_layers=2, n_steps=0, device=dev,
                                cpml_axes="physical")], ids=["tm", "te", "3d"])
def test_a_solve_without_steps_has_a_gradient_of_zero(cuda, make):
    s = make(cuda)
    e = torch.full(s.grid_shape, 2.0, dtype=torch.float64, device=cuda, requires_grad=True)
    r = s.forward(e, source={"type": "gaussian_pulse"})
    (g,) = torch.autograd.grad((r.field.double() ** 2).sum() + r.field.sum(), e)
    assert not r.field.any() and g.shape == e.shape and not g.any()
