"""The tiled design-layer kernels at the edges of their tiles, against the CPU
oracle, and in place."""

from __future__ import annotations

import pytest
import torch

from oracle import design_ref

from conftest import rel_l2



# one layer smaller than the filter's border, tiles of 32 x 64 met exactly and
# missed by one cell, more than one tile each way, 1 and 63 taps
@pytest.mark.gpu
@pytest.mark.parametrize("shape,radius", [((1, 1, 1), 4.0), ((2, 5, 200), 31.0), ((3, 32, 64), 3.0),
                                          ((2, 33, 65), 0.0), ((4, 31, 63), 31.0),
                                          ((1, 97, 129), 31.0)])
def test_tiles_of_the_density_filter(cuda, shape, radius):
    from diffnano_b200.design.projection import density_to_eps
    g = torch.Generator().manual_seed(3)
    rho = torch.rand(shape, generator=g, dtype=torch.float32)
    w = torch.rand(shape, generator=g, dtype=torch.float32)
    x = rho.double().requires_grad_(True)
    ref = design_ref.density_to_eps(x, radius, 2.0, 0.5, "tanh", 1.0, 3.0)
    (ref * w.double()).sum().backward()
    xd = rho.to(cuda).requires_grad_(True)
    out = density_to_eps(xd, radius, 2.0, 0.5, "tanh", 1.0, 3.0)
    (out * w.to(cuda)).sum().backward()
    # two sums of n products round at most 2 (n + 1) times (2^-24 each, the rounded
    # taps included), and the projection's slope and curvature at beta = 2 are
    # below 1.4 and 3; its own tanh is good to a few ulp
    n = 2 * int(radius) + 1
    tol = (2 * (n + 1) * 4.4 + 16) * 2.0 ** -24
    assert rel_l2(out, ref) < tol
    assert rel_l2(xd.grad, x.grad) < tol


@pytest.mark.gpu
def test_density_outputs_may_be_the_input(cuda):
    import ctypes

    from diffnano_b200 import _lib
    g = torch.Generator().manual_seed(4)
    rho = torch.rand(2, 70, 150, generator=g).to(cuda)
    d = _lib.DnDensity(2, 70, 150, 1, 3.0, 4.0, 0.5, 1.0, 3.0)
    work, filt, eps, drho = (torch.empty_like(rho) for _ in range(4))
    f, b = _lib.lib().dn_density_forward, _lib.lib().dn_density_backward
    p = lambda t: t.data_ptr()  # noqa: E731
    s = torch.cuda.current_stream().cuda_stream
    assert f(ctypes.byref(d), p(rho), p(work), p(filt), p(eps), s) == 0
    assert b(ctypes.byref(d), p(filt), p(rho), p(work), p(drho), s) == 0
    a, e = rho.clone(), torch.empty_like(rho)
    assert f(ctypes.byref(d), p(a), p(work), p(a), p(e), s) == 0
    assert torch.equal(a, filt) and torch.equal(e, eps)
    a = rho.clone()
    assert f(ctypes.byref(d), p(a), p(work), p(e), p(a), s) == 0
    assert torch.equal(e, filt) and torch.equal(a, eps)
    a = rho.clone()
    assert b(ctypes.byref(d), p(filt), p(a), p(work), p(a), s) == 0
    assert torch.equal(a, drho)


@pytest.mark.gpu
@pytest.mark.parametrize("shift", [1, 149, 70 * 150, 2 * 70 * 150 - 1])
def test_density_outputs_may_share_memory_with_the_input(cuda, shift):
    """Outputs that begin `shift` values into the input, or before it, and one buffer
    for both outputs (eps is what stays)."""
    import ctypes

    from diffnano_b200 import _lib
    g = torch.Generator().manual_seed(6)
    rho = torch.rand(2, 70, 150, generator=g).to(cuda)
    n = rho.numel()
    d = _lib.DnDensity(2, 70, 150, 1, 3.0, 4.0, 0.5, 1.0, 3.0)
    work, filt, eps, other = (torch.empty_like(rho) for _ in range(4))
    s = torch.cuda.current_stream().cuda_stream

    def run(r, f, e):
        assert _lib.lib().dn_density_forward(ctypes.byref(d), r.data_ptr(), work.data_ptr(),
                                             f.data_ptr(), e.data_ptr(), s) == 0

    run(rho, filt, eps)
    for first, second in ((0, shift), (shift, 0)):
        for swap in (False, True):
            buf = torch.zeros(n + shift, device=cuda)
            r, o = buf[first:first + n], buf[second:second + n]
            r.copy_(rho.reshape(-1))
            run(r, *((other, o) if swap else (o, other)))
            want = (filt, eps) if swap else (eps, filt)
            assert torch.equal(other, want[0]) and torch.equal(o, want[1].reshape(-1))
    run(rho, other, other)
    assert torch.equal(other, eps)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 8, 32), (3, 9, 33), (1, 1, 70), (2, 70, 1)])
def test_blocks_of_the_pools(cuda, shape):
    from diffnano_b200.design import projection as P
    g = torch.Generator().manual_seed(5)
    x0 = torch.randint(0, 3, shape, generator=g).float()   # many ties
    w = torch.randint(-4, 5, shape, generator=g).float()   # sums are exact
    for op in ("erode", "dilate"):
        x = x0.clone().requires_grad_(True)
        ref = getattr(design_ref, op)(x)
        (ref * w).sum().backward()
        xd = x0.to(cuda).requires_grad_(True)
        out = getattr(P, op)(xd)
        (out * w.to(cuda)).sum().backward()
        assert torch.equal(out.cpu(), ref.detach())
        assert torch.equal(xd.grad.cpu(), x.grad)
