"""Where the dissipation increments of a fused stage come from, counted in launches: one for the three axes
on small meshes, three that sum them on larger ones; the line lies by consumer, type and order."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,N,M,launches", [
    (0, 6, (12, 12, 12), 1), (0, 6, (13, 13, 14), 1), (0, 6, (14, 14, 13), 3), (0, 6, (16, 16, 16), 3),
    (1, 6, (16, 16, 16), 1), (0, 4, (16, 16, 40), 1), (0, 5, (33, 32, 32), 3), (1, 4, (41, 40, 40), 3)])
def test_sipg(wt, ctx, prec, N, M, launches):
    g = wt.Mesh.uniform_hex(ctx, N, M, outer_tag=0, precision=prec)
    ws = wt.make_wave3d_workspace(g)
    ws.set_mu(40.0)
    u, v = g.zeros(), g.zeros()
    u += 1.0
    n0 = ctx.launch_count()
    wt.step_rk4_sipg(u, v, ws, 1e-4, 1, tau=40.0, eps_KO=0.1)
    # the first traces, then the increments and the stage itself four times
    assert ctx.launch_count() - n0 == 1 + 4 * (launches + 1)


@pytest.mark.parametrize("N,M,launches", [(4, (16, 16, 16), 1), (4, (16, 16, 17), 3), (8, (10, 10, 10), 1), (8, (11, 10, 10), 3)])
def test_rk4(wt, ctx, N, M, launches):
    g = wt.Mesh.uniform_hex(ctx, N, M, outer_tag=7, warp_A=0.03)
    c, ws = wt.sample_background3d(g, wt.BG_ADM_PERTURBED, wt.workloads.adm_params(3)), wt.make_wave3d_workspace(g)
    ws.set_mu(40.0)
    P, Q = g.zeros(), g.zeros()
    P += 1.0
    n0 = ctx.launch_count()
    wt.step_rk4_curved(P, Q, c, ws, 1e-4, 1, 0.1, wt.make_bc3d([2] * 6), True)
    # two kernels a stage and its increments; n = 8: five fused launches, increments before each
    assert ctx.launch_count() - n0 == (5 + 5 * launches if N == 8 else 8 + 4 * launches)


def test_both_consumers_on_one_workspace(wt, ctx):
    """SIPG steps that split do not make RK4 steps that sum read the split buffer, nor the other way round."""
    import torch
    g = wt.Mesh.uniform_hex(ctx, 4, (16, 16, 40), outer_tag=7)  # split for SIPG, summed for RK4
    c, bc = wt.sample_background3d(g, wt.BG_ADM_PERTURBED, wt.workloads.adm_params(3)), wt.make_bc3d([2] * 6)
    gen = torch.Generator().manual_seed(3)
    P0, Q0 = (torch.rand(g.nn, generator=gen, dtype=torch.float64).cuda() for _ in range(2))

    def rk4(ws):
        P, Q = P0.clone(), Q0.clone()
        wt.step_rk4_curved(P, Q, c, ws, 1e-5, 2, 0.1, bc, True)
        return P, Q

    def sipg(ws):
        u, v = P0.clone(), Q0.clone()
        wt.step_rk4_sipg(u, v, ws, 1e-5, 2, tau=20.0, eps_KO=0.1)
        return u, v

    ws = [wt.make_wave3d_workspace(g) for _ in range(4)]
    alone = rk4(ws[0]), sipg(ws[1])
    after = rk4(ws[2]), sipg(ws[2])
    before = sipg(ws[3]), rk4(ws[3])
    for a, b in ((alone[0], after[0]), (alone[1], after[1]), (alone[0], before[1]), (alone[1], before[0])):
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
