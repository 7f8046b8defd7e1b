"""The masked error norm's fold over the CTAs' partials: fewer partials than the fold's threads, about as
many, and several a thread."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,roots", [(6, 1), (8, 2), (25, 2), (33, 3)])
def test_error_norm_of_a_known_offset(tgh, N, roots):
    case = tgh.gauge_wave_case(eps_ko=0.5)
    f = tgh.gh_forest(case, N, roots)
    P = tgh.GHProblem(case, f, 4, margin_check=False)
    u = P.initial_state(P.statevector(), 0.0)
    # an offset of the same size at every point: L2 = Linf = |offset| over the 20 variables
    d = torch.linspace(1.0, 2.0, 20, dtype=torch.float64, device="cuda")
    u.view(f.nblocks, 20, -1).add_(d[None, :, None])
    want = float(d.norm())
    l2, linf = P.error_norm(u, 0.0)
    # a difference of O(1) values is off by eps, and a sum of n positive terms in any order by less than n eps
    assert abs(l2 / want - 1.0) < 1e-12 and abs(linf / want - 1.0) < 1e-14
    P.close()
