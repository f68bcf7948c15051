"""Boundary terms of the kernels of any order, evaluated face by face: elements with outer faces on
both ends of an axis, edge and corner nodes under different kinds per face (affine form), excised
faces and prescribed data, against the oracle (src/boundaries3d.jl:131-232)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("N,M,metric,kinds,exc", [
    (2, (1, 1, 1), False, [4, 2, 1, 3, 2, 4], 0),
    (4, (1, 3, 9), False, [2, 4, 3, 1, 4, 2], 0),
    (5, (2, 1, 1), True, [4] * 6, 8),
    (6, (3, 1, 2), True, [1] * 6, 8),
    (7, (1, 2, 1), False, [4, 4, 2, 2, 1, 3], 0),
    (7, (1, 1, 2), True, [4] * 6, 0),
])
@pytest.mark.parametrize("f32", [False, True])
def test_face_terms(wt, ctx, O, N, M, metric, kinds, exc, f32):
    import torch
    A = 0.05 if metric else 0.0
    g = wt.Mesh.uniform_hex(ctx, N, M, outer_tag=7, warp_A=A, precision=wt.WT_F32 if f32 else wt.WT_F64)
    o = O.OracleMesh(N, M, A=A, outer_tag=7)
    if exc:
        bd = o.get("bdry").copy()
        bd[4::6][bd[4::6] != 0] = exc
        o.set_bdry(bd)
        g.set_bdry(bd)
    p = wt.workloads.adm_params(N)
    coef, ws = wt.sample_background3d(g, wt.BG_ADM_PERTURBED, p), wt.make_wave3d_workspace(g)
    rng = np.random.default_rng(N)
    d64 = [rng.standard_normal(o.nn).astype(np.float32).astype(np.float64) for _ in range(5)]
    dt_ = torch.float32 if f32 else torch.float64
    dd = [torch.tensor(a, dtype=dt_, device="cuda") for a in d64]
    bc = wt.make_bc3d(kinds, gPhi=dd[0], gPi=dd[1], gDx=dd[2], gDy=dd[3], gDz=dd[4], excision_tag=exc)
    bo = O.make_bc(kinds, gPhi=d64[0], gPi=d64[1], gDx=d64[2], gDy=d64[3], gDz=d64[4], excision_tag=exc)
    x, y, z = o.coords()
    P, Q = (torch.tensor(a, dtype=dt_, device="cuda") for a in (
        np.sin(2.1 * x + 0.3) * np.cos(1.7 * y) * np.sin(2.9 * z + 0.2), np.cos(1.3 * x) * np.sin(2.2 * y + 0.4)))
    dP, dQ = wt.wave3d_curved_rhs(g.empty(), g.empty(), P, Q, coef, ws, 0.0, bc, metric)
    rP, rQ = o.rhs_curved(o.background(2, p), P.double().cpu().numpy(), Q.double().cpu().numpy(), bc=bo,
                          use_metric=metric)
    # one sweep multiplies the roundings by about N^2 M over the field's wavenumber, Pidot takes two
    eps = 6e-8 if f32 else 1.1e-16
    s = 1 + N * N * max(M) / 3.0
    assert rel(dP.double().cpu().numpy(), rP) < 20 * eps * s
    assert rel(dQ.double().cpu().numpy(), rQ) < 20 * eps * s * s
