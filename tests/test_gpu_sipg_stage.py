"""The fused SIPG stage: every order, element counts that leave the last CTA partly empty, Dirichlet
and Sommerfeld faces, with and without dissipation (one launch for the three axes' increments on small
meshes, three on the last case's size), one step (trace kernel first) and several (graph replay)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(2, (7, 3, 1), 0, 0.1, 3), (3, (5, 1, 2), 7, 0.0, 1), (4, (10, 10, 9), 0, 0.1, 1), (5, (3, 2, 2), 7, 0.1, 4),
         (6, (7, 7, 7), 0, 0.0, 3), (7, (2, 3, 1), 7, 0.1, 2), (8, (2, 1, 3), 0, 0.1, 3), (8, (21, 21, 20), 7, 0.1, 1)]


# (the last case's size is for the launch rule, which both types share)
@pytest.mark.parametrize("N,M,tag,eps,steps,f32", [c + (False,) for c in CASES] + [c + (True,) for c in CASES[:-1]])
def test_sipg_stage(wt, ctx, O, N, M, tag, eps, steps, f32):
    import torch
    g = wt.Mesh.uniform_hex(ctx, N, M, outer_tag=tag, precision=wt.WT_F32 if f32 else wt.WT_F64)
    o = O.OracleMesh(N, M, outer_tag=tag)
    ws = wt.make_wave3d_workspace(g)
    x, y, z = o.coords()
    u0 = np.sin(2.1 * x + 0.3) * np.cos(1.7 * y) * np.sin(2.9 * z + 0.2)
    v0 = np.cos(1.3 * x) * np.sin(2.2 * y + 0.4) * np.cos(0.8 * z)
    dt_ = torch.float32 if f32 else torch.float64
    u, v = (torch.tensor(a, dtype=dt_, device="cuda") for a in (u0, v0))
    tau, dt = 1.5 * (N - 1) ** 2, 0.1 * o.min_spacing()
    wt.step_rk4_sipg(u, v, ws, dt, steps, tau=tau, eps_KO=eps)
    ur, vr = o.evolve_sipg(u0, v0, dt, steps, tau=tau, eps_ko=eps)
    # one right-hand side amplifies the rounding of u by about tau N^2 / dx^2 per unit time; u carries dt^2 of it
    eps_ = 6e-8 if f32 else 1.1e-16
    amp = 4 * steps * dt * tau * N * N * max(M) ** 2
    assert np.linalg.norm(u.double().cpu().numpy() - ur) < 40 * eps_ * (1 + dt * amp) * np.linalg.norm(ur)
    assert np.linalg.norm(v.double().cpu().numpy() - vr) < 40 * eps_ * (1 + amp) * (
        np.linalg.norm(vr) + np.linalg.norm(ur))
