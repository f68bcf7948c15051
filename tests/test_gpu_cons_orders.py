"""The conservative right-hand side and RK4 steps of the kernels of any order at every order: element
counts that leave the last CTA partly empty and that change the elements per CTA, the affine and the
curvilinear form, Sommerfeld and full-Dirichlet faces, both types."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


CASES = [(2, (9, 5, 7), 0.0, False, 2), (3, (11, 11, 9), 0.03, True, 4), (4, (1, 2, 1), 0.05, True, 2),
         (4, (11, 9, 9), 0.0, False, 4), (5, (7, 9, 5), 0.05, True, 2), (5, (3, 1, 2), 0.0, False, 2),
         (6, (5, 1, 3), 0.05, True, 4), (6, (7, 7, 7), 0.05, True, 2), (7, (2, 3, 1), 0.05, True, 2),
         (7, (3, 2, 2), 0.0, False, 4), (8, (2, 1, 3), 0.0, False, 2)]


@pytest.mark.parametrize("N,M,A,metric,kind", CASES)
@pytest.mark.parametrize("f32", [False, True])
def test_cons_orders(wt, ctx, O, N, M, A, metric, kind, f32):
    import torch
    g = wt.Mesh.uniform_hex(ctx, N, M, outer_tag=7, warp_A=A, precision=wt.WT_F32 if f32 else wt.WT_F64)
    o = O.OracleMesh(N, M, A=A, outer_tag=7)
    p = wt.workloads.adm_params(N)
    coef, ws = wt.sample_background3d(g, wt.BG_ADM_PERTURBED, p), wt.make_wave3d_workspace(g)
    co, bc, bo = o.background(2, p), wt.make_bc3d([kind] * 6), O.make_bc([kind] * 6)
    x, y, z = o.coords()
    P0 = np.sin(2.1 * x + 0.3) * np.cos(1.7 * y) * np.sin(2.9 * z + 0.2)
    Q0 = np.cos(1.3 * x) * np.sin(2.2 * y + 0.4) * np.cos(0.8 * z)
    dt_ = torch.float32 if f32 else torch.float64
    P, Q = (torch.tensor(a, dtype=dt_, device="cuda") for a in (P0, Q0))
    P64, Q64 = P.double().cpu().numpy(), Q.double().cpu().numpy()
    dP, dQ = wt.wave3d_curved_rhs(g.empty(), g.empty(), P, Q, coef, ws, 0.0, bc, metric)
    rP, rQ = o.rhs_curved(co, P64, Q64, bc=bo, use_metric=metric)
    # Pidot differentiates twice: each sweep multiplies the roundings by about N^2 M over the field's wavenumber
    eps = 6e-8 if f32 else 1.1e-16
    tol = 20 * eps * (1 + (N * N * max(M) / 3.0) ** 2)
    assert rel(dP.double().cpu().numpy(), rP) < 20 * eps * (1 + N * N * max(M) / 3.0)
    assert rel(dQ.double().cpu().numpy(), rQ) < tol
    dt = 0.2 * o.min_spacing() / wt.workloads.max_speed(p)
    wt.step_rk4_curved(P, Q, coef, ws, dt, 4, 0.0, bc, metric)
    sP, sQ = o.evolve_curved(co, P64, Q64, dt, 4, bc=bo, use_metric=metric)
    assert rel(P.double().cpu().numpy(), sP) < tol and rel(Q.double().cpu().numpy(), sQ) < tol
