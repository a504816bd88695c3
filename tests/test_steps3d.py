"""3-D runs as one call of many steps (dependent launches, monitor gradients stored by
the reverse step before) against as many calls of one step (nothing overlaps, each
gradient injected by its own launch): the same bits."""

from __future__ import annotations

import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("shape,n_mon", [((2, 5, 9), 0), ((7, 18, 70), 1), ((40, 17, 33), 2),
                                         ((12, 40, 130), 4)])
def test_one_call_equals_many(cuda, shape, n_mon, dtype):
    from diffnano_b200 import _lib
    from diffnano_b200.solvers import _setup
    from diffnano_b200.solvers._engine import Engine

    T, (D, H, W) = 25, shape
    dl, dt = 20.0, 8.0
    src = {"type": "gaussian_pulse", "spread": 60.0, "t0": 80.0,
           "pos": [D // 2, H // 2, W // 2]}
    g = torch.Generator().manual_seed(41)
    eps = (1.5 + 2.0 * torch.rand(shape, generator=g, dtype=torch.float64)).to(cuda, dtype)
    fields = torch.randn((6, *shape), generator=g, dtype=torch.float64).to(cuda, dtype)
    lam = torch.randn((6, *shape), generator=g, dtype=torch.float64).to(cuda, dtype)

    # monitors that share cells and, the first and the last, a component
    phase = torch.randn((n_mon, T, 2, 2), generator=g, dtype=torch.float64).to(cuda)
    acc, mons = [], (_lib.DnMonitor * max(n_mon, 1))()
    for m in range(n_mon):
        comp = (_lib.DN_EX, _lib.DN_HY, _lib.DN_EZ, _lib.DN_EX)[m]
        lo, hi = [0, m % H, 0], [D, H, max(1, W - m)]
        n = (hi[0] - lo[0]) * (hi[1] - lo[1]) * (hi[2] - lo[2])
        acc.append(torch.randn((2, n, 2), generator=g, dtype=torch.float64).to(cuda))
        mons[m].component, mons[m].n_freq, mons[m].n_t = comp, 2, T
        mons[m].phase, mons[m].acc = phase[m].data_ptr(), acc[m].data_ptr()
        for a in range(3):
            mons[m].box.lo[a], mons[m].box.hi[a] = lo[a], hi[a]

    def run(per_call):
        eng = Engine(is3d=True, shape=shape, dl=dl, dt=dt, pml_layers=1, dtype=dtype,
                     device=cuda, n_steps=T, wave=_setup.waveform_table(T, dt, 0.1, src),
                     src_box=_setup.source_box_3d(shape, src), src_comp=_lib.DN_EZ,
                     axes=_lib.DN_AXES_PHYSICAL)
        eng.set_eps(eps)
        eng._ws = torch.empty(0, dtype=torch.uint8, device=cuda)  # launch by launch
        eng.A[..., :W] = fields
        buf = eng.curl_buffer(T)
        rec = eng.curl_record(buf, 0, T)
        for t in range(0, T, per_call):
            eng.run(t, per_call, record=rec)
        la, lb = torch.zeros_like(eng.A), torch.zeros_like(eng.A)
        la[..., :W] = lam
        grad = torch.zeros((D, H, eng.Wp), dtype=torch.float64, device=cuda)
        for t in range(T, 0, -per_call):
            if eng.adjoint(la, lb, rec, grad, mons if n_mon else None, n_mon, t, per_call):
                la, lb = lb, la
        eng.check_status()
        return (eng.B if eng.cur_b else eng.A)[..., :W], la[..., :W], grad[..., :W]

    for a, b in zip(run(T), run(1)):
        assert float(a.abs().max()) > 0
        assert torch.equal(a, b)
