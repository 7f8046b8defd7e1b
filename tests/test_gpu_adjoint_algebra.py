"""The reverse sweep of the point algebra: the transpose identity <lam, J v> = <J^T lam, v> against the
tangent-linear form, over the gauge sources, the interior variants, the orders and no dissipation."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = {
    "none": lambda t: t.gauge_wave_case(eps_ko=0.5, gamma0=1.0, gamma2=-0.5),
    "none_plain": lambda t: t.gauge_wave_case(eps_ko=0.0, gamma0=0.0, gamma2=0.0),
    "sampled": lambda t: t.shifted_minkowski_case(eps_ko=0.5, gamma0=1.0, gamma2=-0.5),
    "algebraic_layer": lambda t: t.kerr_schild_case(a=0.7, halfwidth=2.0, gauge="algebraic"),
    "sampled_layer": lambda t: t.kerr_schild_case(a=0.7, halfwidth=2.0, gauge="sampled", gamma2=0.3),
    "frozen": lambda t: t.kerr_schild_case(a=0.7, halfwidth=2.0, gauge="algebraic", variant="frozen"),
}


@pytest.mark.parametrize("q,N", [(2, 9), (4, 8), (8, 11)])
@pytest.mark.parametrize("name", sorted(CASES))
def test_reverse_sweep_is_the_transpose_of_the_tangent(tgh, name, q, N):
    case = CASES[name](tgh)
    f = tgh.gh_forest(case, N, 2)
    P = tgh.GHProblem(case, f, q, margin_check=False)
    g = torch.Generator(device="cuda").manual_seed(7)

    def rand():
        return torch.randn(P.state_length, dtype=torch.float64, device="cuda", generator=g)

    u = P.initial_state(P.statevector(), 0.1) + 1e-4 * rand()
    v, lam = rand(), rand()
    du, dut = torch.zeros_like(u), torch.zeros_like(u)
    lam_u, th = P.adjoint_rhs(u, 0.1, lam)
    P.tangent_rhs(du, dut, u, v, 0.1, "state")
    a, b = float(torch.dot(lam, dut)), float(torch.dot(lam_u, v))
    # both sides are sums of L terms of size |lam| |J v|; each term's rounding is eps times a few thousand
    # operations, and the sums' roundings add like a random walk
    bound = 1e-12 * float(lam.norm() * dut.norm())
    assert abs(a - b) <= bound, (a, b, bound)
    if case.interior:
        zero = torch.zeros_like(u)
        for k, direction in enumerate(("rho_max", "ramp", "damp_near")):
            P.tangent_rhs(du, dut, u, zero, 0.1, direction)
            a = float(torch.dot(lam, dut))
            assert abs(a - th[k]) <= 1e-12 * float(lam.norm() * dut.norm()) + 1e-300, (direction, a, th[k])
    P.close()
