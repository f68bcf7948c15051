"""The buffers that only make steps faster (the fused stages' second flux buffer, the dissipation
increments of all axes): held by whole-step calls alone, found again after set_fused, and left out where
the device's memory is short, with the results of the steps that have them."""
import pytest

pytestmark = pytest.mark.gpu


def _solve(wt, ctx, M, prec, eps=0.0):
    import torch
    g = wt.Mesh.uniform_hex(ctx, 8, M, outer_tag=7, warp_A=0.05, precision=prec)
    c = wt.sample_background3d(g, wt.BG_ADM_PERTURBED, wt.workloads.adm_params(3))
    ws = wt.make_wave3d_workspace(g)
    if eps:
        ws.set_mu(40.0)
    gen = torch.Generator().manual_seed(1)
    P, Q = (torch.rand(g.nn, generator=gen, dtype=torch.float64).to(g.dtype).cuda() for _ in range(2))
    bc = wt.make_bc3d([2] * 6)

    def step():
        n0 = ctx.launch_count()
        wt.step_rk4_curved(P, Q, c, ws, 1e-4, 1, eps, bc, True)
        return ctx.launch_count() - n0

    return g, c, ws, P, Q, bc, step


def test_batch_and_sipg_hold_no_second_flux_buffer(wt, ctx):
    g, c, ws, P, Q, bc, _ = _solve(wt, ctx, 4, wt.WT_F32)
    field = 4 * g.nn
    live = ctx.memory()[0]
    b = wt.Batch(ctx)
    b.add(P, Q, c, ws, 1e-4, bc)
    b.step(1)
    # stages 3, accumulators 2, low parts 2, copy of the high part 1 (the flux came with the workspace)
    assert ctx.memory()[0] - live < 9 * field
    b.close()
    g = wt.Mesh.uniform_hex(ctx, 8, 4, outer_tag=0, precision=wt.WT_F32)
    ws = wt.make_wave3d_workspace(g)
    live = ctx.memory()[0]
    wt.step_rk4_sipg(g.zeros(), g.zeros(), ws, 1e-4, 1)
    # the same and two sets of face traces, 0.75 each
    assert ctx.memory()[0] - live < 10.5 * field


@pytest.mark.parametrize("prec", [0, 1])
def test_fused_stages_after_two_kernel_ones(wt, ctx, prec):
    *_, ws, _, _, _, step = _solve(wt, ctx, (3, 2, 2), prec)
    ws.set_fused(False)
    assert step() == 8
    ws.set_fused(True)
    assert step() == 5


def test_steps_where_memory_is_short(wt, ctx):
    import torch
    made = [_solve(wt, ctx, 3, wt.WT_F32), _solve(wt, ctx, 3, wt.WT_F64, 0.1),
            _solve(wt, ctx, 3, wt.WT_F32), _solve(wt, ctx, 3, wt.WT_F64, 0.1)]
    for s in made:
        wt.wave3d_curved_rhs(s[0].empty(), s[0].empty(), s[3], s[4], s[1], s[2], 0.0, s[5], True)
    free, total = torch.cuda.mem_get_info()
    assert free > total // 4
    fill = torch.empty(free - total // 48, dtype=torch.uint8, device="cuda")
    try:
        # two-kernel stages; the increments summed axis by axis: three launches a stage
        assert made[0][6]() == 8 and made[1][6]() == 8 + 12
    finally:
        del fill
        torch.cuda.empty_cache()
    # five launches; one each for the increments of the first stage, between the stages and of the last Pi
    assert made[2][6]() == 5 and made[3][6]() == 5 + 5
    assert torch.equal(made[0][3], made[2][3]) and torch.equal(made[0][4], made[2][4])
    for k in (3, 4):  # the increments' sum rounds in another order: a few units of the last place of a step's change
        assert (made[1][k] - made[3][k]).norm() <= 1e-13 * made[3][k].norm()
    made[0][2].set_fused(True)
    assert made[0][6]() == 5
