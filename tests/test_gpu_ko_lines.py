"""The line-local Kreiss-Oliger kernel at the edges of its launch rules: every order, lines of one
element, open and closed, lines that change the pencils per CTA (512 threads) and that need the
1024-thread instantiation, and the longest line it takes (longer ones: six apply_D! passes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(2, (3, 1, 2), False), (3, (2, 5, 1), True), (4, (32, 2, 1), False), (4, (33, 1, 1), False),
         (5, (1, 1, 21), True), (6, (15, 1, 2), False), (7, (11, 2, 1), False), (8, (9, 1, 1), True),
         (8, (1, 65, 1), False), (8, (1, 1, 128), False), (7, (1, 147, 1), False)]


@pytest.mark.parametrize("N,M,periodic", CASES)
@pytest.mark.parametrize("f32", [False, True])
def test_ko_lines(wt, ctx, O, N, M, periodic, f32):
    import torch
    g = wt.Mesh.uniform_hex(ctx, N, M, periodic=periodic, outer_tag=7, warp_A=0.0 if periodic else 0.03,
                            precision=wt.WT_F32 if f32 else wt.WT_F64)
    o = O.OracleMesh(N, M, A=0.0 if periodic else 0.03, periodic=periodic, outer_tag=7)
    ws = wt.make_wave3d_workspace(g)
    ws.set_mu(float(o.mu()))
    f = np.random.default_rng(N).standard_normal(o.nn)
    dt = torch.float32 if f32 else torch.float64
    ft = torch.tensor(f, dtype=dt, device="cuda")
    out = wt.ko_add(g.zeros(), ft, 0.1, ws).double().cpu().numpy()
    ref = np.zeros(o.nn)
    o.ko_add(ref, ft.double().cpu().numpy(), 0.1 * (1.0 / o.mu()) ** 5)
    # white noise does not cancel in D: each of the six passes adds a few N roundings of its operands'
    # size, |D| |D^-1| amplified at most by the ratio of a pass's largest entry to its norm (< N)
    eps = 6e-8 if f32 else 1.1e-16
    assert np.linalg.norm(out - ref) < 6 * 2 * N * N * eps * np.linalg.norm(ref)
