"""The batched form computes a point that same-level leaves share once (RhsArgs' PointRun) and reads it back
for every copy: the plain form, which computes every copy, gives the same bits - on one periodic block that is
its own neighbour, on meshes whose blocks keep all, some or none of their upper faces, with odd edges, and
across refinement faces, where a face stays when the leaf beyond is of another level."""
import pytest
import torch

from helpers import two_level_forest

pytestmark = pytest.mark.gpu

MESHES = {
    "one_block": lambda t: (t.gauge_wave_case(eps_ko=0.5, gamma0=1.0), lambda c: t.gh_forest(c, 11, 1), 4),
    "periodic_q2": lambda t: (t.gauge_wave_case(eps_ko=0.5, gamma0=1.0), lambda c: t.gh_forest(c, 9, 2), 2),
    "periodic_n32": lambda t: (t.gauge_wave_case(eps_ko=0.5, gamma0=1.0), lambda c: t.gh_forest(c, 32, 2), 4),
    "half_periodic": lambda t: (t.shifted_minkowski_case(eps_ko=0.5, gamma0=1.0), lambda c: t.gh_forest(c, 8, 3), 4),
    "hole_n16_q6": lambda t: (t.kerr_schild_case(a=0.7, halfwidth=3.0), lambda c: t.gh_forest(c, 16, 3), 6),
    "hole_n32": lambda t: (t.kerr_schild_case(a=0.7, halfwidth=4.0), lambda c: t.gh_forest(c, 32, 3), 4),
    "two_level": lambda t: (t.gauge_wave_case(eps_ko=0.5, gamma0=1.0), lambda c: two_level_forest(t, c, N=8), 4),
    "moving_levels_n8": lambda t: (t.kerr_schild_case(a=0.7, v=0.1, halfwidth=4.0, gauge="algebraic"),
                                   lambda c: t.hole_forest(c, 8, 4, [2.0, 1.6]), 4),
    "moving_levels_n32": lambda t: (t.kerr_schild_case(a=0.7, v=0.1, halfwidth=6.0, gauge="algebraic"),
                                    lambda c: t.hole_forest(c, 32, 2, [1.6]), 4),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", sorted(MESHES))
def test_batched_form_gives_every_copy_the_plain_forms_bits(tgh, name, precision):
    case, forest, q = MESHES[name](tgh)
    f = forest(case)
    P = tgh.GHProblem(case, f, q, margin_check=False, precision=precision)
    g = torch.Generator(device="cuda").manual_seed(5)
    u = P.initial_state(P.statevector(), 0.0)
    u += 1e-6 * torch.randn(u.shape, dtype=torch.float64, device="cuda", generator=g)
    P.settle(u, 0.0)
    dt = 0.25 * f.h0 / 2 ** int(f.level.max()) / 4
    a, b = u.clone(), u.clone()
    P.step_batched(a, 0.0, dt, 1)
    P.rk4_step(b, 0.0, dt)
    assert torch.isfinite(a).all()
    assert torch.equal(a, b), float((a - b).abs().max())
    P.close()
