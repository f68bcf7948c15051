"""FP32 SIPG stepping (wt_step_rk4_sipg) depends on (u, ut) alone: nothing of an earlier call stays in
the workspace, whether the caller steps the same arrays again or refills them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,steps,eps", [(4, 1, 0.0), (6, 4, 0.1), (8, 3, 0.0)])
def test_refilled_arrays_step_like_fresh_ones(wt, ctx, N, steps, eps):
    import torch
    g = wt.Mesh.uniform_hex(ctx, N, (3, 2, 2), outer_tag=0, precision=wt.WT_F32)
    ws = wt.make_wave3d_workspace(g)
    dt, tau = 0.1 * g.min_spacing(), 1.5 * (N - 1) ** 2
    gen = torch.Generator().manual_seed(N)
    a0, b0 = (torch.randn(g.nn, generator=gen).cuda() for _ in range(2))

    def step(u, v, w):
        wt.step_rk4_sipg(u, v, w, dt, steps, tau=tau, eps_KO=eps)
        return u.clone(), v.clone()

    u, v = a0.clone(), b0.clone()
    first = step(u, v, ws)
    # the same arrays, zeroed: the zero state is a fixed point
    u.zero_(), v.zero_()
    z = step(u, v, ws)
    assert not z[0].any() and not z[1].any()
    # refilled with a state 1e6 times smaller: the bits of a workspace never stepped before
    u.copy_(1e-6 * a0), v.copy_(1e-6 * b0)
    small = step(u, v, ws)
    fresh = step(1e-6 * a0, 1e-6 * b0, wt.make_wave3d_workspace(g))
    assert torch.equal(small[0], fresh[0]) and torch.equal(small[1], fresh[1])
    # refilled with the first state
    u.copy_(a0), v.copy_(b0)
    again = step(u, v, ws)
    assert torch.equal(again[0], first[0]) and torch.equal(again[1], first[1])
    # n steps in one call and in n calls
    u.copy_(a0), v.copy_(b0)
    for _ in range(steps):
        wt.step_rk4_sipg(u, v, ws, dt, 1, tau=tau, eps_KO=eps)
    assert torch.equal(u, first[0]) and torch.equal(v, first[1])
