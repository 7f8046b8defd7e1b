"""The batched form computes a point that same-level leaves share once (RhsArgs' PointRun) and reads it back
for every copy: the plain form, which computes every copy, gives the same bits - on one periodic block that is
its own neighbour, on meshes whose blocks keep all, some or none of their upper faces, with odd edges, and
across refinement faces, where a face stays when the leaf beyond is of another level, around a vertex whose
computed copy is three moves away in only one order of the axes, and across a periodic wrap beside a Dirichlet
boundary, whose values differ by rounding between the two faces."""
from dataclasses import replace

import numpy as np
import pytest
import torch

from helpers import two_level_forest

pytestmark = pytest.mark.gpu



def refined_roots(tgh, case, N, refined):
    """2^3 root blocks, those at the root coordinates `refined` replaced by their eight children."""
    f = tgh.gh_forest(case, N, 2)
    leaves = []
    for c in f.corner:
        if tuple(int(v) // N for v in c) in refined:
            leaves += [(1, tuple(int(2 * c[d]) + o[d] * N for d in range(3))) for o in np.ndindex(2, 2, 2)]
        else:
            leaves.append((0, tuple(int(v) for v in c)))
    leaves.sort()
    return tgh.Forest(N, f.lo, f.h0, f.cells0, f.periodic, np.array([l for l, _ in leaves], dtype=np.int32),
                      np.array([c for _, c in leaves], dtype=np.int32))


def wave(tgh, periodic, A=0.05, d=1.0):
    return replace(tgh.gauge_wave_case(A=A, eps_ko=0.5, gamma0=1.0), background={"kind": "gauge_wave", "A": A, "d": d},
                   periodic=periodic)


# the same-level leaves around the centre are (0, 0, 0), (0, 1, 0), (1, 1, 0), (1, 1, 1) and an axis permutation of
# them: from the first to the last the moves are y, x, z (z, y, x)
STAIRS = {"yxz": {(1, 0, 0), (0, 0, 1), (0, 1, 1), (1, 0, 1)}, "zyx": {(1, 0, 0), (0, 1, 0), (1, 1, 0), (1, 0, 1)},
          "xzy": {(0, 1, 0), (0, 0, 1), (0, 1, 1), (1, 1, 0)}}

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
    **{f"stairs_{k}": lambda t, r=r: (wave(t, (False,) * 3), lambda c: refined_roots(t, c, 8, r), 4)
       for k, r in STAIRS.items()},
    "wrap_beside_dirichlet": lambda t: (wave(t, (True, False, True), 0.4, 1 / 3), lambda c: t.gh_forest(c, 8, 2), 4),
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
