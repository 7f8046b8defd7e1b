"""The working array after a batched step: its owned points are the returned state's at every copy of a shared point,
those the step left out (a block's upper faces) among them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def owned(work, f, q):
    n1, G = f.N + 1, q // 2 + 1
    W = n1 + 2 * G
    return work.view(f.nblocks, 20, W, W, W)[:, :, G:G + n1, G:G + n1, G:G + n1].reshape(-1)


@pytest.mark.parametrize("name", ["periodic", "static_hole", "moving_levels"])
def test_owned_points_are_the_state(tgh, name):
    q, N = 4, 8
    if name == "periodic":
        case = tgh.gauge_wave_case(eps_ko=0.5, gamma0=1.0)
        f = tgh.gh_forest(case, N, 2)
    elif name == "static_hole":
        case = tgh.kerr_schild_case(a=0.7, halfwidth=2.0)
        f = tgh.gh_forest(case, N, 3)
    else:
        case = tgh.kerr_schild_case(a=0.7, v=0.1, halfwidth=4.0, gauge="algebraic")
        f = tgh.hole_forest(case, N, 4, [2.0, 1.6])
    P = tgh.GHProblem(case, f, q, margin_check=False)
    g = torch.Generator(device="cuda").manual_seed(7)
    u = P.initial_state(P.statevector(), 0.0)
    u += 1e-6 * torch.randn(u.shape, dtype=torch.float64, device="cuda", generator=g)
    P.settle(u, 0.0)
    dt = 0.25 * f.h0 / 2 ** int(f.level.max()) / 4
    for n in range(2):
        P.step_batched(u, n * dt, dt, 1)
        w = P.copy_work()
        assert torch.equal(owned(w, f, q), u)
        # a range of blocks sees the same points
        b0, nb = f.nblocks // 2, f.nblocks - f.nblocks // 2
        assert torch.equal(P.copy_work_blocks(b0, nb), w.view(f.nblocks, -1)[b0:].reshape(-1))
    # after a prepare the array holds that fill as it is: every copy its primary's value, as settle returns it (where
    # levels meet a step leaves the copies apart)
    v = u.clone()
    P.settle(v, 2 * dt)
    P.prepare(u, 2 * dt)
    assert torch.equal(owned(P.copy_work(), f, q), v)
    du, ref = torch.zeros_like(u), torch.zeros_like(u)
    P.rhs(du, 2 * dt)
    P.gh_rhs(ref, u, 2 * dt)
    assert torch.equal(du, ref)
    P.close()
