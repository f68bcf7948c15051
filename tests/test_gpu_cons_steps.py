"""Four RK4 steps of the kernels of any order, by their increments: what the steps add to the state against
what the oracle's add, so that a lost step or a wrong stage weight shows in FP32 too, where the bound on
one right-hand side (tests of the conservative orders) is as large as the whole change of Phi."""
import numpy as np
import pytest

CASES = [(2, (9, 5, 7), 0.0, False, 2), (3, (11, 11, 9), 0.03, True, 4), (4, (1, 2, 1), 0.05, True, 2),
         (4, (11, 9, 9), 0.0, False, 4), (5, (7, 9, 5), 0.05, True, 2), (6, (5, 1, 3), 0.05, True, 4),
         (6, (7, 7, 7), 0.05, True, 2), (7, (2, 3, 1), 0.05, True, 2), (8, (2, 1, 3), 0.0, False, 2)]
STEPS = 4


def setup(W, O, N, M, A, kind):
    o = O.OracleMesh(N, M, A=A, outer_tag=7)
    p = W.adm_params(N)
    x, y, z = o.coords()
    P0 = (np.sin(2.1 * x + 0.3) * np.cos(1.7 * y) * np.sin(2.9 * z + 0.2)).astype(np.float32).astype(np.float64)
    Q0 = (np.cos(1.3 * x) * np.sin(2.2 * y + 0.4) * np.cos(0.8 * z)).astype(np.float32).astype(np.float64)
    return o, p, P0, Q0, o.background(2, p), O.make_bc([kind] * 6), 0.2 * o.min_spacing() / W.max_speed(p)


def bounds(o, co, bo, N, M, metric, P0, Q0, dt, eps):
    """What rounding may add: a derivative's roundings are N^2 M / 3 times those of its operand, Pi-dot takes
    two, and 20 eps covers a right-hand side's sums; Phi-dot passes Pi's error on (lapse and shift below 2);
    the state itself is rounded at every step."""
    rP, rQ = (np.linalg.norm(r) for r in o.rhs_curved(co, P0, Q0, bc=bo, use_metric=metric))
    s, t = 1 + N * N * max(M) / 3.0, STEPS * dt
    tQ = t * 20 * eps * s * s * rQ + 2 * STEPS * eps * np.linalg.norm(Q0)
    tP = t * 20 * eps * s * rP + 2 * t * tQ + 2 * STEPS * eps * np.linalg.norm(P0)
    return tP, tQ


@pytest.mark.gpu
@pytest.mark.parametrize("N,M,A,metric,kind", CASES)
@pytest.mark.parametrize("f32", [False, True])
def test_increments(wt, ctx, O, N, M, A, metric, kind, f32):
    import torch
    o, p, P0, Q0, co, bo, dt = setup(wt.workloads, O, N, M, A, kind)
    g = wt.Mesh.uniform_hex(ctx, N, M, outer_tag=7, warp_A=A, precision=wt.WT_F32 if f32 else wt.WT_F64)
    coef, ws = wt.sample_background3d(g, wt.BG_ADM_PERTURBED, p), wt.make_wave3d_workspace(g)
    P, Q = (torch.tensor(a, dtype=g.dtype, device="cuda") for a in (P0, Q0))
    wt.step_rk4_curved(P, Q, coef, ws, dt, STEPS, 0.0, wt.make_bc3d([kind] * 6), metric)
    sP, sQ = o.evolve_curved(co, P0, Q0, dt, STEPS, bc=bo, use_metric=metric)
    tP, tQ = bounds(o, co, bo, N, M, metric, P0, Q0, dt, 6e-8 if f32 else 1.1e-16)
    assert np.linalg.norm(P.double().cpu().numpy() - sP) < tP
    assert np.linalg.norm(Q.double().cpu().numpy() - sQ) < tQ


def mistaken(o, co, bo, metric, P0, Q0, dt, which):
    """The oracle's steps with a mistake planted: the last step left out, or its last stage weighted as a
    middle one."""
    P, Q = o.evolve_curved(co, P0, Q0, dt, STEPS - 1, bc=bo, use_metric=metric)
    if which == "step":
        return P, Q
    f = lambda a, b: o.rhs_curved(co, a, b, bc=bo, use_metric=metric)
    k1 = f(P, Q)
    k2 = f(P + 0.5 * dt * k1[0], Q + 0.5 * dt * k1[1])
    k3 = f(P + 0.5 * dt * k2[0], Q + 0.5 * dt * k2[1])
    k4 = f(P + dt * k3[0], Q + dt * k3[1])
    return tuple(y + dt / 6 * (a + 2 * b + 2 * c + 2 * d) for y, a, b, c, d in zip((P, Q), k1, k2, k3, k4))


@pytest.mark.parametrize("which", ["step", "weight"])
def test_bounds_tell_mistakes(O, which):
    """(CPU) the bounds are well below what the mistakes change: a step in both fields, a weight in Phi."""
    from conftest import load_package
    for N, M, A, metric, kind in CASES:
        o, p, P0, Q0, co, bo, dt = setup(load_package().workloads, O, N, M, A, kind)
        sP, sQ = o.evolve_curved(co, P0, Q0, dt, STEPS, bc=bo, use_metric=metric)
        mP, mQ = mistaken(o, co, bo, metric, P0, Q0, dt, which)
        tP, tQ = bounds(o, co, bo, N, M, metric, P0, Q0, dt, 6e-8)
        assert np.linalg.norm(mP - sP) > 3 * tP, (N, M)
        assert which == "weight" or np.linalg.norm(mQ - sQ) > 3 * tQ, (N, M)
