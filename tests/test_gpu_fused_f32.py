"""GPU: the compensated FP32 n = 8 stages (gradient half, divergence half, both
fused) against each other and against the oracle.

The halves and the fused stage are instantiations of one kernel, so a fused step
and one of two-kernel stages must agree bit for bit.  Against the FP64 oracle
(wave3d_curved_rhs!, src/wave3d_curved.jl:205-258, and classic RK4) the state,
initially the rounded oracle state, may be off by FP32 rounding: 2^-24 = 6e-8 of
the initial data and of each step's increment, amplified by the divergence's
(n - 1)^2 / h ~ 1e2 in Pi at most, hence 1e-5.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL32 = 1e-5


def f32(a):
    return np.asarray(a, dtype=np.float32).astype(np.float64)


def rel(a, b):
    a = np.asarray(a, dtype=np.float64)
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _run(wt, ctx, g, c, Phi, Pi, dt, nsteps, bc, fused):
    import torch
    ws = wt.make_wave3d_workspace(g)
    ws.set_fused(fused)
    P = torch.tensor(Phi, dtype=torch.float32, device="cuda")
    Q = torch.tensor(Pi, dtype=torch.float32, device="cuda")
    wt.step_rk4_curved(P, Q, c, ws, dt, 1, bc3d=bc, metric=True)
    n0 = ctx.launch_count()
    wt.step_rk4_curved(P, Q, c, ws, dt, 1, bc3d=bc, metric=True)
    launches = ctx.launch_count() - n0
    wt.step_rk4_curved(P, Q, c, ws, dt, nsteps - 2, bc3d=bc, metric=True)
    ctx.synchronize()
    assert not ctx.nonfinite()
    return P, Q, launches


@pytest.mark.parametrize("M,kinds,periodic,exc", [
    (1, [2] * 6, False, 0),            # one element, every face an outer face
    ((5, 2, 3), [2] * 6, False, 0),    # fewer elements than SMs
    ((10, 9, 9), [4] * 6, False, 0),   # more than the resident CTAs; full-Dirichlet data
    ((3, 4, 2), [1] * 6, False, 8),    # characteristic data, -z faces excised
    (3, None, True, 0),                # every face a SAT face
])
def test_fused_f32(wt, ctx, O, M, kinds, periodic, exc):
    import torch
    tag = 0 if periodic else 7
    g = wt.Mesh.uniform_hex(ctx, 8, M, periodic=periodic, outer_tag=tag, warp_A=0.05, precision=wt.WT_F32)
    o = O.OracleMesh(8, M, A=0.05, periodic=periodic, outer_tag=tag)
    if exc:
        bd = o.get("bdry").copy()
        bd[4::6][bd[4::6] != 0] = exc
        o.set_bdry(bd)
        g.set_bdry(bd)
    p = wt.workloads.adm_params(5)
    x, y, z = o.coords()
    Phi = wt.workloads.gaussian_field(x, y, z, *wt.workloads.pulses(5, 3))
    Pi = 0.2 * np.sin(2 * np.pi * x) * Phi
    dt = 0.2 * o.min_spacing() / wt.workloads.max_speed(p)
    c = wt.sample_background3d(g, 2, p)
    bc = None if kinds is None else wt.make_bc3d(kinds, excision_tag=exc)
    Pf, Qf, lf = _run(wt, ctx, g, c, Phi, Pi, dt, 7, bc, True)
    Pu, Qu, lu = _run(wt, ctx, g, c, Phi, Pi, dt, 7, bc, False)
    assert (lf, lu) == (5, 8)
    assert torch.equal(Pf, Pu) and torch.equal(Qf, Qu)
    obc = None if kinds is None else O.make_bc(kinds, excision_tag=exc)
    Po, Qo = o.evolve_curved(o.background(2, p), *map(f32, (Phi, Pi)), dt, 7, bc=obc, use_metric=True)
    assert rel(Pf.double().cpu().numpy(), Po) < TOL32
    assert rel(Qf.double().cpu().numpy(), Qo) < TOL32
