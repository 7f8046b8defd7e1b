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


# the interior kernel's points a CTA on 8 blocks around the hole and 148 SMs: 128 up to 11^3, 256 at 13^3, 512 from 16^3
@pytest.mark.parametrize("N", [11, 13, 16])
@pytest.mark.parametrize("variant,v", [("damped", 0.0), ("damped", 0.1), ("frozen", 0.0)])
def test_interior_on_small_meshes(tgh, oracle, N, variant, v):
    case = tgh.kerr_schild_case(a=0.7, v=v, halfwidth=2.0, variant=variant, gauge="algebraic")
    # the bound of the right-hand side's parity everywhere
    assert _rhs_error(tgh, oracle, case, tgh.gh_forest(case, N, 2), 4, 0.3) < 1e-12
