"""Where the dissipation increments of a fused stage come from: one launch for the three axes on meshes of
up to 2^19 nodes, three that sum them on larger ones."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,launches", [((12, 12, 12), 1), ((13, 13, 14), 1), ((14, 14, 13), 3), ((16, 16, 16), 3)])
def test_ko_split(wt, ctx, M, launches):
    g = wt.Mesh.uniform_hex(ctx, 6, M, outer_tag=0)
    ws = wt.make_wave3d_workspace(g)
    ws.set_mu(40.0)
    u, v = g.zeros(), g.zeros()
    u += 1.0
    n0 = ctx.launch_count()
    wt.step_rk4_sipg(u, v, ws, 1e-4, 1, tau=40.0, eps_KO=0.1)
    # the first traces, then the increments and the stage itself four times
    assert ctx.launch_count() - n0 == 1 + 4 * (launches + 1)
