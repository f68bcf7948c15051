"""Launch variants of a batch's generic groups: the autotuner chooses among different CTA shapes only (none
to choose from n = 6 up), and the shapes that orders 2 to 5 have give the same bits."""
import pytest

pytestmark = pytest.mark.gpu


def _member(wt, ctx, b, N, M, seed):
    import torch
    g = wt.Mesh.uniform_hex(ctx, N, M, outer_tag=7, warp_A=0.05)
    c = wt.sample_background3d(g, wt.BG_ADM_PERTURBED, wt.workloads.adm_params(seed))
    ws = wt.make_wave3d_workspace(g)
    gen = torch.Generator().manual_seed(seed)
    P, Q = (torch.rand(g.nn, generator=gen, dtype=torch.float64).cuda() for _ in range(2))
    return b.add(P, Q, c, ws, 1e-4, wt.make_bc3d([2] * 6)), P, Q, ws


def test_autotuner_leaves_single_shapes_alone(wt, ctx):
    b = wt.Batch(ctx)
    keep = [_member(wt, ctx, b, N, 7, N) for N in (4, 5, 6, 7)]
    for k in range(6):  # each change of membership tunes anew
        slot, *rest = _member(wt, ctx, b, 4, 2, 20 + k)
        b.step(1)
        choice = {g[0]: (g[3] & 3, g[3] >> 2) for g in b.groups()}
        assert choice[6] == (0, 0) and choice[7] == (0, 0)
        assert max(choice[5]) <= 1 and max(choice[4]) <= 2
        b.remove(slot)
    b.close()
    del keep


@pytest.mark.parametrize("N,M", [(2, 17), (3, 11), (4, 9), (5, 8)])
def test_shapes_give_the_same_bits(wt, ctx, N, M):
    import torch
    out = []
    for var in (0, 1, 2):
        b = wt.Batch(ctx)
        b.set_variant(var, var)
        _, P, Q, ws = _member(wt, ctx, b, N, M, 5)
        b.step(3)
        out.append((P, Q))
        b.close()
    for P, Q in out[1:]:
        assert torch.equal(P, out[0][0]) and torch.equal(Q, out[0][1])
