"""The strong-form right-hand side at every order: the last CTA partly empty, Sommerfeld, Dirichlet and
excised faces, warped elements, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M,tag", [(2, (5, 4, 1), 7), (3, (3, 3, 1), 0), (4, (5, 1, 1), 7), (5, (3, 1, 1), 8),
                                     (6, (2, 1, 3), 0), (7, (2, 2, 1), 7), (8, (1, 3, 2), 0)])
@pytest.mark.parametrize("f32", [False, True])
def test_strong_orders(wt, ctx, O, N, M, tag, f32):
    import torch
    g = wt.Mesh.uniform_hex(ctx, N, M, outer_tag=tag, warp_A=0.04, precision=wt.WT_F32 if f32 else wt.WT_F64)
    o = O.OracleMesh(N, M, A=0.04, outer_tag=tag)
    ws = wt.make_wave3d_workspace(g)
    rng = np.random.default_rng(N)
    dt = torch.float32 if f32 else torch.float64
    u, v = (torch.tensor(rng.standard_normal(o.nn), dtype=dt, device="cuda") for _ in range(2))
    out = wt.wave_strong_rhs_mesh(g.empty(), u, v, ws, sommerfeld_R=3.0)
    ref = o.rhs_strong(u.double().cpu().numpy(), v.double().cpu().numpy(), R=3.0)
    # FP64 arithmetic in both types: two sweeps of N-term sums (and of the metric's derivative), each within
    # N roundings of operands that white noise does not cancel; FP32 rounds the result once more
    tol = 4 * N * N * 1.1e-16 * 10 + (6e-8 if f32 else 0.0)
    err = np.linalg.norm(out.double().cpu().numpy() - ref) / np.linalg.norm(ref)
    assert err < tol
