"""The surrogate's readout at the edges of its row groups, and its gradients, against
FP64 sums of the same BF16 inputs."""

from __future__ import annotations

import pytest
import torch

from conftest import rel_l2


# fewer rows than a group, groups and remainders, fewer and more columns than a warp's
# 128, one column group; odd widths take the scalar form
@pytest.mark.gpu
@pytest.mark.parametrize("nb,H,W,C", [(1, 1, 4, 1), (2, 3, 132, 3), (1, 17, 60, 8), (3, 34, 256, 5),
                                      (2, 33, 35, 4)])
def test_readout_and_its_gradients(cuda, nb, H, W, C):
    from diffnano_b200 import _lib
    g = torch.Generator().manual_seed(H * W)
    x = torch.randn(nb, C, H, W, generator=g).to(torch.bfloat16).to(cuda)
    dR = torch.randn(nb, W, C, generator=g).to(torch.bfloat16).to(cuda)
    r = torch.randn(H, C, generator=g).to(cuda)
    out = torch.empty(nb, W, C, dtype=torch.bfloat16, device=cuda)
    dx = torch.empty_like(x)
    dr = torch.empty(nb, H, C, device=cuda)
    s = torch.cuda.current_stream().cuda_stream
    L, p = _lib.lib(), lambda t: t.data_ptr()
    assert L.dn_fno_readout(p(x), p(r), nb, H, W, C, p(out), s) == 0
    assert L.dn_fno_readout_bwd(p(x), p(r), p(dR), nb, H, W, C, p(dx), p(dr), s) == 0
    X, D, Rr = x.double(), dR.double(), r.double()
    # sums of n terms in FP32, against the sum of their absolute values; BF16 outputs
    # round once more (2^-9 of the value)
    def close(got, ref, mag, n, bf16):
        tol = (n + 1) * 2.0 ** -24 * mag + (2.0 ** -8 * ref.abs() if bf16 else 0.0)
        assert bool(((got.double() - ref).abs() <= tol + 1e-30).all())

    close(out, torch.einsum("hc,bchw->bwc", Rr, X),
          torch.einsum("hc,bchw->bwc", Rr.abs(), X.abs()), H, True)
    ref = torch.einsum("hc,bwc->bchw", Rr, D)
    close(dx, ref, ref.abs(), 1, True)
    close(dr, torch.einsum("bwc,bchw->bhc", D, X),
          torch.einsum("bwc,bchw->bhc", D.abs(), X.abs()), W, False)
    # one output at a time: the same values
    only = torch.empty_like(dr)
    assert L.dn_fno_readout_bwd(p(x), p(r), p(dR), nb, H, W, C, None, p(only), s) == 0
    assert torch.equal(only, dr)
    assert rel_l2(dx.double(), ref) < 2.0 ** -8
