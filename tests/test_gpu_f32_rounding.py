"""Rounding of the compensated FP32 n = 8 divergence on a flux that oscillates within an element: the
error against the FP64 kernels is that of plain FP32 sums (numpy, fused multiply-adds) of the rounded
flux.  A line of elements of unit size, flat background: Pi-dot = D D Phi along x."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M = 64


def fma(a, b, c):
    return (np.float64(a) * np.float64(b) + np.float64(c)).astype(np.float32)


def divergence(F, G, H):
    """D F with the centred-flux SAT, periodic line, F [M, 8]: 0.5 G by plain sums, doubled."""
    Gh, c = (0.5 * G).astype(np.float32), 1.0 / (2.0 * H[0])
    w = (F[:, :1] * Gh[:, 0]).astype(np.float32)
    for p in range(1, 8):
        w = fma(F[:, p:p + 1], Gh[:, p], w)
    w = np.float32(2) * w
    jump = F - np.roll(F[:, ::-1], 1, axis=0)  # [:, 0]: value minus the left neighbour's last
    w[:, 0] = fma(np.float32(c), jump[:, 0], w[:, 0])
    w[:, 7] = fma(np.float32(c), np.roll(F[:, 0], -1) - F[:, 7], w[:, 7])
    return w


@pytest.mark.parametrize("waves", [61, 40])
def test_divergence_rounding(wt, ctx, waves):
    import torch
    bc = None
    mesh, coef, ws = {}, {}, {}
    for prec in (wt.WT_F64, wt.WT_F32):
        mesh[prec] = wt.Mesh.uniform_hex(ctx, 8, (M, 1, 1), 0.0, float(M), periodic=True, precision=prec)
        coef[prec] = wt.sample_background3d(mesh[prec], wt.BG_MINKOWSKI)
        ws[prec] = wt.make_wave3d_workspace(mesh[prec])
    x, H, G = wt.gll_operators(8)
    X = np.arange(M)[:, None] + x
    rng = np.random.default_rng(waves)
    e = e0 = 0.0
    for _ in range(20):
        line = np.sin(2 * np.pi * (waves / M * X + rng.random())).astype(np.float32)
        u = torch.tensor(np.broadcast_to(line[:, None, :], (M, 64, 8)).reshape(-1).copy(), device="cuda")
        d = {}
        for prec, t in ((wt.WT_F64, torch.float64), (wt.WT_F32, torch.float32)):
            P = u.to(t)
            _, dQ = wt.wave3d_curved_rhs(mesh[prec].empty(), mesh[prec].empty(), P, torch.zeros_like(P), coef[prec],
                                         ws[prec], 0.0, bc, True)
            d[prec] = dQ.double().cpu().numpy().reshape(M, 64, 8)[:, 0]
        g = [mesh[wt.WT_F64].empty() for _ in range(3)]
        wt.apply_gradient3d(*g, u.double(), ws[wt.WT_F64])
        F = g[0].cpu().numpy().reshape(M, 64, 8)[:, 0].astype(np.float32)
        e += float(np.sum((d[wt.WT_F32] - d[wt.WT_F64]) ** 2))
        e0 += float(np.sum((divergence(F, G, H).astype(np.float64) - d[wt.WT_F64]) ** 2))
    # beyond the flux's rounding the kernel's gradient has two more, of half the flux's size at most
    assert e <= 1.15 ** 2 * e0, np.sqrt(e / e0)
