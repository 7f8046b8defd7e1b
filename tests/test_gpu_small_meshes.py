"""Kernels whose launch depends on the number of CTAs, at mesh sizes on either side of the lines, against the oracle."""
import numpy as np
import pytest
import torch

from helpers import rhs_error, rhs_scale

pytestmark = pytest.mark.gpu


def _rhs_error(tgh, oracle, case, f, q, t, precision="fp64"):
    P = tgh.GHProblem(case, f, q, margin_check=False, precision=precision, tuned=False)
    O = oracle.problem(case, f, q)
    u = O.initial_state(O.statevector(), t) + tgh.perturbation(f, amplitude=1e-6, seed=11)
    ref = np.zeros(O.L)
    O.gh_rhs(ref, u, t)
    du = torch.full((O.L,), float("nan"), dtype=torch.float64, device="cuda")
    P.gh_rhs(du, torch.from_numpy(u).cuda(), t)
    err = rhs_error(du.cpu().numpy(), ref, rhs_scale(O.work(), f, q), f)
    P.close()
    return err


# the interior kernel's points a CTA around the hole and 148 SMs: on 8 blocks 128 up to 15^3 and 512 from 16^3 on, where
# one block of 27 holds the sphere 128 up to 32^3 and 512 at 33^3
@pytest.mark.parametrize("N,roots,halfwidth", [(11, 2, 2.0), (15, 2, 2.0), (16, 2, 2.0), (32, 3, 4.0), (33, 3, 4.0)])
@pytest.mark.parametrize("variant,v", [("damped", 0.0), ("damped", 0.1), ("frozen", 0.0)])
def test_interior_on_small_meshes(tgh, oracle, N, roots, halfwidth, variant, v):
    case = tgh.kerr_schild_case(a=0.7, v=v, halfwidth=halfwidth, variant=variant, gauge="algebraic")
    # the bound of the right-hand side's parity everywhere
    assert _rhs_error(tgh, oracle, case, tgh.gh_forest(case, N, roots), 4, 0.3) < 1e-12


# the one-point Pi kernel's registers: a block's launch is below the line (27 CTAs), the mesh's of 1,688 above it
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("q", [2, 4, 6, 8])
@pytest.mark.parametrize("eps", [0.5, 0.0])
def test_register_bounds_give_the_same_bits(tgh, q, precision, eps):
    case = tgh.gauge_wave_case(eps_ko=eps, gamma0=1.0)
    P = tgh.GHProblem(case, tgh.gh_forest(case, 14, 4), q, margin_check=False, precision=precision, tuned=False)
    if precision == "fp64":
        P.set_variant(pi="l1")
    u = P.initial_state(P.statevector(), 0.0)
    u += 1e-6 * torch.randn(u.shape, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    P.settle(u, 0.0)
    a, b = u.clone(), u.clone()
    P.rk4_step(a, 0.0, 1e-3)
    P.rk4_step_blocks(b, 0.0, 1e-3)
    assert torch.isfinite(a).all() and torch.equal(a, b)
    P.close()


# the batched form below the line (138 CTAs of runs) against the oracle
@pytest.mark.parametrize("q", [2, 4, 6, 8])
def test_batched_step_on_a_small_mesh(tgh, oracle, q):
    case = tgh.gauge_wave_case(eps_ko=0.5, gamma0=1.0)
    f = tgh.gh_forest(case, 12, 2)
    P = tgh.GHProblem(case, f, q, margin_check=False, tuned=False)
    O = oracle.problem(case, f, q)
    u = O.initial_state(O.statevector(), 0.0) + tgh.perturbation(f, amplitude=1e-6, seed=11)
    a = torch.from_numpy(u).cuda()
    P.settle(a, 0.0)  # the copies of a shared point agree: the batched form starts from the primaries
    u = a.cpu().numpy()
    dt = 0.25 * f.h0 / 4
    P.step_batched(a, 0.0, dt, 1)
    O.rk4_step(u, 0.0, dt)
    assert np.abs(a.cpu().numpy() - u).max() < 1e-12  # the parity bound of a step on states of order one
    P.close()
